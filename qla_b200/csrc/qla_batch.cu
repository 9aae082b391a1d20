// qla_batch.cu -- many fields of uneven volume, each running its own short
// sequence of level-1 operations, in one persistent launch.
//
// A lattice code often applies a short level-1 sequence to many independent
// fields (sub-lattices, sources, time slices).  Launching QLA's functions
// once per field and step costs a launch each and leaves the GPU idle on the
// small fields.  Here a plan cuts every field into tiles of 32 sites and deals
// the tiles to the warps of one persistent launch, in contiguous runs of equal
// estimated cost.  Each field carries a small program (qlagpu_F3_batch_program):
// streams (its record arrays, some gathered through an int32 index) and steps
// drawn from the engine's per-site operators -- colour-matrix left
// multiplication (lmult_site), spin projection and reconstruction (the
// SpprojOp / SpreconOp bodies), real multiples and copies -- so a field's
// results are bit-identical to the separate QLA_F3 calls the steps stand for.
//
// Every warp runs by itself, with no block-wide synchronisation: it brings the
// next tile's records into shared memory while it computes the present one
// (bulk copies; gathered V and M records, whose length no bulk copy takes,
// with cp.async), and the index tile of the tile after that.  Then each lane
// takes one site through the field's steps.  Every value a step reads or makes
// (stream records, registers, stored results) has a fixed shared-memory slot,
// chosen by the planner, so a step is one call of a routine compiled for its
// operation and record kinds, chosen by a uniform switch, with nothing kept in
// registers between steps.  Stored results leave by one bulk store per stream.
// Partial tiles and fields whose arrays are only 8-B aligned run the same
// steps with 8-B copies.
//
// The launch (qlagpu_batch_run) passes only the plan's device table: it can
// be replayed from a captured CUDA graph.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <type_traits>
#include <vector>

#include "../../include/qla_b200_runtime.h"
#include "qla_launch.cuh"
#include "qla_ops.cuh"

namespace qlab {

constexpr int kMaxStreams = 8, kMaxSteps = 8, kMaxFields = 1024;
constexpr int kReg0 = 8, kReg1 = 9;
enum BKind : int { BK_V = 0, BK_H = 1, BK_D = 2, BK_M = 3 };
enum BRole : int { BR_IN = 0, BR_OUT = 1, BR_INOUT = 2 };
enum BOp : int { BOP_LMULT = 0, BOP_SPPROJ = 1, BOP_SPRECON = 2, BOP_RTIMES = 3, BOP_COPY = 4 };
// complex numbers per V, H, D, M record (F3)
__host__ __device__ constexpr int kncplx(int kind) { return kind == BK_V ? 3 : kind == BK_H ? 6 : kind == BK_D ? 12 : 9; }

struct BStream {
  char* base;
  const int* idx;
  int kind, role;
  unsigned lim;       // gathered: indices must lie in [0, lim); 0: unchecked
  int wide;           // records start on 16-B boundaries
  int used;           // some step reads it (IN / INOUT: it is copied in)
  unsigned slot;      // IN / INOUT: its records' place in the stage
  unsigned idx_slot;  // gathered: three index tiles in the warp's fixed area
  unsigned out;       // OUT / INOUT: the stored result's place in the stage
};
struct BStep {
  int code;  // StepCode
  int eqop, mu, sign;
  unsigned a, b, old, res;  // places in the stage of the operands, of the value that peq / meq update, and of the result
  float r;
  int pad;
};

struct alignas(16) BField {
  BStream s[kMaxStreams];
  BStep st[kMaxSteps];
  int nstreams, nsteps;
  long long n, tile0;
  int bulk;            // every contiguous array that is read or written starts on a 16-B boundary
  unsigned tx;         // bytes the contiguous streams of a full tile bring
  int ngather;         // gathered streams that some step reads
  int gather[kMaxStreams];
};

struct BatchParams {
  const BField* fields;
  const long long* start;  // first tile of each run, and the end; block b takes runs b, b + grid, ...
  int runs;
  int nfields;
  unsigned fixed_bytes, stage_bytes, warp_bytes;
  int stages;              // 1 or 2
  unsigned* err;
};

struct BatchPlan {
  BField* dfields;    // device: the field table, then the runs' first tiles
  long long* dstart;
  int nfields, threads, grid, stages, runs;
  long long ntiles;
  unsigned fixed_bytes, stage_bytes, warp_bytes;
  size_t smem;
};

// The routine of a step: LMULT by the kind of b and the adjoints, then the
// other operations by their record kind.
enum StepCode : int { SC_LMULT = 0, SC_SPPROJ = 16, SC_SPRECON = 17, SC_RTIMES = 20, SC_COPY = 24 };

constexpr int kDescWords = (int)((sizeof(BField) + 15) / 16);  // 16-B words

// bytes of one record, and of its shared slot
__host__ __device__ constexpr unsigned rec_b(int kind) { return (unsigned)kncplx(kind) * 8u; }


// --- copies between global memory and a warp's slots with plain instructions:
// partial tiles, and fields that are not 16-B aligned
__device__ __forceinline__ void run_in(unsigned char* dst, const char* src, unsigned bytes, int lane) {
#pragma unroll 1
  for (unsigned o = lane * 8u; o < bytes; o += 256u) cp_async_8(dst + o, src + o);
}
__device__ __forceinline__ void run_out(char* dst, const unsigned char* src, unsigned bytes, int lane) {
#pragma unroll 1
  for (unsigned o = lane * 8u; o < bytes; o += 256u)
    *reinterpret_cast<uint2*>(dst + o) = *reinterpret_cast<const uint2*>(src + o);
}
// a gathered tile: P 8-B pieces per record, 32 / P records at a time, one lane
// per piece (a lane keeps its piece number, so its addresses advance by
// constants); nv records, record r at index idx[r]; the records of the lanes in
// `bad` read zero
template <int P>
__device__ __forceinline__ void gather_pieces(unsigned char* dst, const char* base, const int* idx, int nv,
                                              unsigned bad, int lane) {
  constexpr int G = 32 / P, ITS = (32 + G - 1) / G;
  const int r0 = lane / P, pc = lane - r0 * P;
  if (r0 >= G) return;
  const char* from = base + pc * 8;
  dst += (r0 * P + pc) * 8;
  idx += r0;
  if (nv == 32 && bad == 0u) {
#pragma unroll
    for (int it = 0; it < ITS; it++)
      if ((it + 1) * G <= 32 || r0 < 32 - it * G)
        cp_async_8(dst + it * G * P * 8, from + (long long)idx[it * G] * (P * 8));
  } else {
#pragma unroll 1
    for (int it = 0; it < ITS; it++) {
      const int r = it * G + r0;
      if (r >= nv) break;
      if ((bad >> r) & 1u)
        *reinterpret_cast<uint2*>(dst + it * G * P * 8) = make_uint2(0u, 0u);
      else
        cp_async_8(dst + it * G * P * 8, from + (long long)idx[it * G] * (P * 8));
    }
  }
}

// --- one record of this lane, in its slot
template <int N>
__device__ __forceinline__ void ld_slot(Cx<float> (&x)[N], const unsigned char* p) {
  load_rec<float, N>(x, p);
}
template <int N>
__device__ __forceinline__ void st_slot(unsigned char* p, const Cx<float> (&y)[N]) {
  store_rec_smem<float, N>(p, y);
}

// (a destination that no eqop reads is zeroed: left undefined, each routine's
// array would stay live around the step loop and the kernel take 255 registers)
template <int N>
__device__ __forceinline__ void zero_slot(Cx<float> (&x)[N]) {
#pragma unroll
  for (int e = 0; e < N; e++) x[e] = Cx<float>{0.f, 0.f};
}

// this lane's record of kind K at place `off` of the stage
struct Slots {
  unsigned char* stage;
  int lane;
  template <int K>
  __device__ __forceinline__ unsigned char* at(unsigned off) const {
    return stage + off + (unsigned)lane * rec_b(K);
  }
};
// A step's result may take the place of a value that has been read for the
// last time, of another record length: every lane has its operands in
// registers before any lane stores.
template <int K, int N>
__device__ __forceinline__ void put(const Slots& sl, unsigned off, const Cx<float> (&y)[N]) {
  __syncwarp();
  st_slot(sl.at<K>(off), y);
  __syncwarp();
}

// --- the steps (the engine's per-site operators).  The eqop is uniform: it is
// branched on once per step, outside the element loops.
template <int K, bool ADJA, bool ADJB>
__device__ __forceinline__ void step_lmult(const BStep& S, const Slots& sl) {
  constexpr int NCOL = K == BK_V ? 1 : K == BK_H ? 2 : K == BK_D ? 4 : 3, N = 3 * NCOL;
  const bool load = (S.eqop == PEQ || S.eqop == MEQ);
  Cx<float> a[9], b[N], y[N];
  ld_slot(a, sl.at<BK_M>(S.a));
  ld_slot(b, sl.at<K>(S.b));
  if (load) ld_slot(y, sl.at<K>(S.old));
  else zero_slot(y);
  // y (0, or the old value) plus or minus a b
  if (S.eqop == EQ || S.eqop == PEQ)
    lmult_site<float, 3, NCOL, ADJA, ADJB>(PEQ, true, a, b, y);
  else
    lmult_site<float, 3, NCOL, ADJA, ADJB>(MEQ, true, a, b, y);
  put<K>(sl, S.res, y);
}
// F's body for (mu, sign), its eqop known at compile time where it is the usual one
template <class F, int LA, int LY>
__device__ __forceinline__ void step_spin(const BStep& S, const Cx<float> (&a)[LA], Cx<float> (&y)[LY]) {
  if (S.eqop == EQ)
    mu_sign_dispatch<F>(S.mu, S.sign, (int)EQ, a, y);
  else if (S.eqop == PEQ)
    mu_sign_dispatch<F>(S.mu, S.sign, (int)PEQ, a, y);
  else
    mu_sign_dispatch<F>(S.mu, S.sign, S.eqop, a, y);
}
__device__ __forceinline__ void step_spproj(const BStep& S, const Slots& sl) {
  Cx<float> a[12], y[6];
  ld_slot(a, sl.at<BK_D>(S.a));
  if (S.eqop == PEQ || S.eqop == MEQ) ld_slot(y, sl.at<BK_H>(S.old));
  else zero_slot(y);
  step_spin<SpprojOp<float, 3>::Body>(S, a, y);
  put<BK_H>(sl, S.res, y);
}
__device__ __forceinline__ void step_sprecon(const BStep& S, const Slots& sl) {
  Cx<float> h[6], y[12];
  ld_slot(h, sl.at<BK_H>(S.a));
  if (S.eqop == PEQ || S.eqop == MEQ) ld_slot(y, sl.at<BK_D>(S.old));
  else zero_slot(y);
  step_spin<SpreconOp<float, 3>::Body>(S, h, y);
  put<BK_D>(sl, S.res, y);
}
template <int K, bool RTIMES>  // RTimesOp, CopyOp
__device__ __forceinline__ void step_map(const BStep& S, const Slots& sl) {
  constexpr int N = kncplx(K);
  Cx<float> b[N], y[N];
  ld_slot(b, sl.at<K>(S.a));
  if (S.eqop == PEQ || S.eqop == MEQ) ld_slot(y, sl.at<K>(S.old));
  else zero_slot(y);
#pragma unroll
  for (int e = 0; e < N; e++) {
    const float pr = RTIMES ? rmul(S.r, b[e].re) : b[e].re, pi = RTIMES ? rmul(S.r, b[e].im) : b[e].im;
    switch (S.eqop) {
      case EQ: y[e].re = pr; y[e].im = pi; break;
      case EQM: y[e].re = -pr; y[e].im = -pi; break;
      case PEQ: y[e].re = radd(y[e].re, pr); y[e].im = radd(y[e].im, pi); break;
      default: y[e].re = rsub(y[e].re, pr); y[e].im = rsub(y[e].im, pi); break;
    }
  }
  put<K>(sl, S.res, y);
}

__device__ __forceinline__ void run_step(const BStep& S, const Slots& sl) {
  switch (S.code) {
    case SC_LMULT + BK_V * 4 + 0: step_lmult<BK_V, false, false>(S, sl); break;
    case SC_LMULT + BK_V * 4 + 2: step_lmult<BK_V, true, false>(S, sl); break;
    case SC_LMULT + BK_H * 4 + 0: step_lmult<BK_H, false, false>(S, sl); break;
    case SC_LMULT + BK_H * 4 + 2: step_lmult<BK_H, true, false>(S, sl); break;
    case SC_LMULT + BK_D * 4 + 0: step_lmult<BK_D, false, false>(S, sl); break;
    case SC_LMULT + BK_D * 4 + 2: step_lmult<BK_D, true, false>(S, sl); break;
    case SC_LMULT + BK_M * 4 + 0: step_lmult<BK_M, false, false>(S, sl); break;
    case SC_LMULT + BK_M * 4 + 1: step_lmult<BK_M, false, true>(S, sl); break;
    case SC_LMULT + BK_M * 4 + 2: step_lmult<BK_M, true, false>(S, sl); break;
    case SC_LMULT + BK_M * 4 + 3: step_lmult<BK_M, true, true>(S, sl); break;
    case SC_SPPROJ: step_spproj(S, sl); break;
    case SC_SPRECON: step_sprecon(S, sl); break;
    case SC_RTIMES + BK_V: step_map<BK_V, true>(S, sl); break;
    case SC_RTIMES + BK_H: step_map<BK_H, true>(S, sl); break;
    case SC_RTIMES + BK_D: step_map<BK_D, true>(S, sl); break;
    case SC_RTIMES + BK_M: step_map<BK_M, true>(S, sl); break;
    case SC_COPY + BK_V: step_map<BK_V, false>(S, sl); break;
    case SC_COPY + BK_H: step_map<BK_H, false>(S, sl); break;
    case SC_COPY + BK_D: step_map<BK_D, false>(S, sl); break;
    default: step_map<BK_M, false>(S, sl); break;
  }
}

// --- a warp's pipeline over the tiles of one field

// What a lane does for the whole field: lane j issues the bulk copies of
// stream j (contiguous input, and result) of full tiles.
struct LaneStream {
  const char* in;         // next tile's records, or nullptr
  char* out;              // this tile's place in the result array, or nullptr
  unsigned bytes;         // 32 records
  unsigned slot, out_slot;
};

// index tile t (32 sites from 32 t) of every gathered stream, into ring place q
__device__ __forceinline__ void fetch_indices(const BField& F, unsigned char* area, unsigned t, unsigned q, int nv,
                                              int lane) {
  if (lane >= nv) return;
  for (int g = 0; g < F.ngather; g++) {
    const BStream& S = F.s[F.gather[g]];
    cp_async_4(area + S.idx_slot + q * 128u + (unsigned)lane * 4u, S.idx + (size_t)t * 32u + lane);
  }
}

// records of tile t (nv sites) of every stream that a step reads (its index
// tile has landed in ring place q): contiguous streams of a full tile by one
// bulk copy each, lane j issuing stream j's; gathered H and D records by one
// bulk copy per lane; gathered V and M records (24 and 72 B: no 16-B multiple
// at 8-B steps) in 8-B pieces.  The stage's barrier gets one arrival with the
// bytes to come.
__device__ __forceinline__ void fetch_tile(const BField& F, LaneStream& L, unsigned char* area, unsigned char* stage,
                                           uint64_t* bar, unsigned t, unsigned q, int nv, unsigned nw, int lane,
                                           unsigned* err) {
  unsigned tx = 0;
  if (F.bulk && nv == 32) {
    tx = F.tx;
    if (L.in) {
      bulk_g2s(stage + L.slot, L.in, L.bytes, bar, policy_evict_first());
      L.in += (size_t)nw * L.bytes;
    }
  } else {
    for (int j = 0; j < F.nstreams; j++) {
      const BStream& S = F.s[j];
      const unsigned rb = rec_b(S.kind);
      if (S.used && !S.idx) run_in(stage + S.slot, S.base + (size_t)t * 32u * rb, (unsigned)nv * rb, lane);
    }
  }
  for (int g = 0; g < F.ngather; g++) {
    const BStream& S = F.s[F.gather[g]];
    const int* idx = reinterpret_cast<const int*>(area + S.idx_slot + q * 128u);
    const int k = lane < nv ? idx[lane] : 0;
    const bool ok = S.lim == 0u || (unsigned)k < S.lim || lane >= nv;
    const unsigned bad = ~__ballot_sync(0xffffffffu, ok);
    if (!ok) raise_dev_error(err, QLA_DEVERR_BAD_INDEX);
    unsigned char* dst = stage + S.slot;
    if (S.wide && (S.kind == BK_D || S.kind == BK_H)) {
      const unsigned rb = rec_b(S.kind);
      if (lane < nv) {
        if (ok) {
          bulk_g2s(dst + lane * rb, S.base + (long long)k * (int)rb, rb, bar, policy_evict_normal());
        } else {
          for (unsigned o = 0; o < rb; o += 16u) *reinterpret_cast<uint4*>(dst + lane * rb + o) = make_uint4(0, 0, 0, 0);
        }
      }
      tx += rb * (unsigned)(nv - __popc(bad));
    } else {
      switch (S.kind) {
        case BK_V: gather_pieces<3>(dst, S.base, idx, nv, bad, lane); break;
        case BK_H: gather_pieces<6>(dst, S.base, idx, nv, bad, lane); break;
        case BK_D: gather_pieces<12>(dst, S.base, idx, nv, bad, lane); break;
        default: gather_pieces<9>(dst, S.base, idx, nv, bad, lane); break;
      }
    }
  }
  if (lane == 0) {
    if (tx)
      mbar_arrive_expect_tx(bar, tx);
    else
      mbar_arrive(bar);
  }
}

// A warp's shared memory: [two stage barriers | field descriptor | index
// tiles (fixed_bytes) | one or two stages].
__global__ void __launch_bounds__(128, 4) batch_program_kernel(const BatchParams p) {
  overlap_begin();
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned nw = blockDim.x >> 5;
  unsigned char* mine = smem + (size_t)warp * p.warp_bytes;
  uint64_t* bar = reinterpret_cast<uint64_t*>(mine);
  uint4* desc = reinterpret_cast<uint4*>(mine + 16);
  unsigned char* area = reinterpret_cast<unsigned char*>(desc + kDescWords);
  unsigned char* stages = area + p.fixed_bytes;
  const BField& F = *reinterpret_cast<const BField*>(desc);
  if (lane == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init_fence();
  }
  unsigned cnt = 0;  // tiles fetched: stage cnt & 1, parity (cnt >> 1) & 1
  bool alive = true;
  for (int run = blockIdx.x; run < p.runs && alive; run += gridDim.x) {
    // a run's tiles are dealt to the block's warps one by one
    long long g = p.start[run] + warp;
    const long long gend = p.start[run + 1];
    if (g >= gend) continue;
    int f;
    {
      int lo = 0, hi = p.nfields - 1;  // last field with tile0 <= g
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (p.fields[mid].tile0 <= g)
          lo = mid;
        else
          hi = mid - 1;
      }
      f = lo;
    }
    for (; g < gend && alive; f++) {
      const uint4* src = reinterpret_cast<const uint4*>(p.fields + f);
      for (int k = lane; k < kDescWords; k += 32) desc[k] = ld_in(src + k);
      __syncwarp();
      const long long ntf = (F.n + 31) / 32;  // tiles of this field (an empty field has none)
      const int ntail = (int)(F.n & 31);      // sites of a partial last tile
      unsigned t = (unsigned)(g - F.tile0 < ntf ? g - F.tile0 : ntf);  // (a warp may skip a small field)
      const unsigned tend = (unsigned)(gend - F.tile0 < ntf ? gend - F.tile0 : ntf);
      auto sites = [&](unsigned u) { return (ntail && (long long)u + 1 == ntf) ? ntail : 32; };
      if (g < F.tile0 + tend) g += ((F.tile0 + tend - g + nw - 1) / nw) * nw;  // this warp's first tile behind it
      if (t < tend) {
        LaneStream L{nullptr, nullptr, 0u, 0u, 0u};
        if (lane < F.nstreams) {
          const BStream& S = F.s[lane];
          L.bytes = 32u * rec_b(S.kind);
          L.slot = S.slot;
          L.out_slot = S.out;
          char* at = S.base + (size_t)t * L.bytes;
          if (S.used && !S.idx) L.in = at;
          if (S.role != BR_IN) L.out = at;
        }
        // fill the pipeline: indices of two tiles, records of the first.  The
        // last results of the field or run before may still be leaving the
        // stage (in a one-stage plan it is the one filled now, and the tile loop
        // waits for them only when it has another tile to fetch): every lane
        // waits until its bulk stores have read their slots, then all go on
        unsigned q = 0;  // ring place of tile t's indices
        fetch_indices(F, area, t, 0, sites(t), lane);
        bulk_wait_read<0>();
        cp_async_wait_all();
        __syncwarp();
        // stage and barrier of the c-th tile this warp fetches, and its parity
        auto place = [&](unsigned c) { return p.stages == 2 ? c & 1u : 0u; };
        auto parity = [&](unsigned c) { return (p.stages == 2 ? c >> 1 : c) & 1u; };
        fetch_tile(F, L, area, stages + place(cnt) * p.stage_bytes, &bar[place(cnt)], t, 0, sites(t), nw, lane, p.err);
        if (t + nw < tend) fetch_indices(F, area, t + nw, 1, sites(t + nw), lane);
        for (; t < tend; t += nw, cnt++) {
          cp_async_wait_all();
          bulk_wait_read<0>();  // the previous tile's results have left their slots
          if (!mbar_wait_bounded(&bar[place(cnt)], parity(cnt), p.err)) alive = false;
          alive = __all_sync(0xffffffffu, alive);
          if (!alive) break;
          // this tile's records and the next tile's indices have landed; a lane's
          // cp.async copies and zeroed records show to the others only behind this
          // barrier (a vote does not order memory)
          __syncwarp();
          const unsigned q1 = q == 2u ? 0u : q + 1u, q2 = q1 == 2u ? 0u : q1 + 1u;
          unsigned char* stage = stages + place(cnt) * p.stage_bytes;
          if (p.stages == 2 && t + nw < tend)
            fetch_tile(F, L, area, stages + (~cnt & 1u) * p.stage_bytes, &bar[~cnt & 1u], t + nw, q1, sites(t + nw), nw,
                       lane, p.err);
          if (t + 2 * nw < tend) fetch_indices(F, area, t + 2 * nw, q2, sites(t + 2 * nw), lane);
          q = q1;
          const int nv = sites(t);
          // (the lanes behind a partial tile compute on what lies in their slots;
          // nothing of it is stored)
          const Slots sl{stage, lane};
          for (int k = 0; k < F.nsteps; k++) run_step(F.st[k], sl);
          // orders this lane's reads and writes of the slots before the async
          // proxy: the bulk stores below and the next bulk copies into the stage
          fence_proxy_async_smem();
          __syncwarp();
          if (F.bulk && nv == 32) {
            if (L.out) {
              bulk_s2g(L.out, stage + L.out_slot, L.bytes,
                       policy_evict_first());
              bulk_commit();
              L.out += (size_t)nw * L.bytes;
            }
          } else {
            for (int j = 0; j < F.nstreams; j++) {
              const BStream& S = F.s[j];
              const unsigned rb = rec_b(S.kind);
              if (S.role != BR_IN)
                run_out(S.base + (size_t)t * 32u * rb, stage + S.out,
                        (unsigned)nv * rb, lane);
            }
            // the result slots are free: this lane's reads of them come before
            // the bulk copies that fill them next
            fence_proxy_async_smem();
            __syncwarp();
          }
          if (p.stages == 1 && t + nw < tend) {
            bulk_wait_read<0>();
            __syncwarp();
            fetch_tile(F, L, area, stages, bar, t + nw, q, sites(t + nw), nw, lane, p.err);
          }
        }
      }
      __syncwarp();  // every lane is done with this field's descriptor
    }
  }
  // a wait that gave up: wait (bounded) once more for the copies of both
  // stages before the warp's shared memory can be released
  if (!alive) {
    for (int s = 0; s < p.stages; s++)
      if (!mbar_wait_bounded(&bar[p.stages == 2 ? (cnt + s) & 1u : 0u], (p.stages == 2 ? (cnt + s) >> 1 : cnt) & 1u,
                             p.err, 200000000ull) &&
          lane == 0)
        raise_dev_error(p.err, QLA_DEVERR_BULK_TIMEOUT);
    cp_async_wait_all();
  }
  bulk_wait_all<0>();
}

// ---------------------------------------------------------------------------
// host side: validation, stage layout, plan

static bool plan_error(const char* who, int f, int k, const char* what) {
  char msg[160];
  if (k >= 0)
    std::snprintf(msg, sizeof msg, "field %d, step %d: %s", f, k, what);
  else
    std::snprintf(msg, sizeof msg, "field %d: %s", f, what);
  set_error(QLAGPU_ERR_ARG, who, msg);
  return false;
}

static bool aligned(const void* p, unsigned a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

// Checks one program and fills its device descriptor: kinds, step codes and
// the shared-memory slots of everything the steps read and make.  Returns
// false with the sticky error set when the program is malformed.
static bool build_field(const char* who, int f, const qlagpu_F3_batch_program& q, BField& b, unsigned& fixed_bytes,
                        unsigned& stage_bytes, long long& cost) {
  std::memset(&b, 0, sizeof(b));
  if (q.n < 0 || q.nstreams < 0 || q.nstreams > kMaxStreams || q.nsteps < 1 || q.nsteps > kMaxSteps)
    return plan_error(who, f, -1, "need n >= 0, 0..8 streams and 1..8 steps");
  b.nstreams = q.nstreams;
  b.nsteps = q.nsteps;
  b.n = q.n;
  for (int j = 0; j < q.nstreams; j++) {
    const qlagpu_batch_stream& s = q.stream[j];
    BStream& d = b.s[j];
    if (s.kind < 0 || s.kind > 3 || s.role < 0 || s.role > 2)
      return plan_error(who, f, -1, "stream kind or role out of range");
    if (!s.base && q.n > 0) return plan_error(who, f, -1, "NULL stream base");
    if (s.index && s.role != BR_IN) return plan_error(who, f, -1, "only IN streams may gather through an index");
    if (s.index && s.nsrc < 0) return plan_error(who, f, -1, "nsrc < 0");
    if (!aligned(s.base, 8) || (s.index && !aligned(s.index, 4)))
      return plan_error(who, f, -1, "stream base must be 8-B aligned and an index 4-B aligned");
    d.base = static_cast<char*>(s.base);
    d.idx = s.index;
    d.lim = s.index ? (unsigned)(s.nsrc < 0x7fffffffLL ? s.nsrc : 0x80000000LL) : 0u;
    d.kind = s.kind;
    d.role = s.role;
    d.wide = aligned(s.base, 16) ? 1 : 0;
  }
  b.bulk = 1;
  int regkind[2] = {-1, -1}, kind_a[kMaxSteps], kind_r[kMaxSteps], load_stream[kMaxSteps];
  int store_step[kMaxStreams];
  for (int j = 0; j < kMaxStreams; j++) store_step[j] = -1;
  auto opnd_kind = [&](int ref, int& kind) -> const char* {
    if (ref == kReg0 || ref == kReg1) {
      kind = regkind[ref - kReg0];
      return kind < 0 ? "operand register read before any step wrote it" : nullptr;
    }
    if (ref < 0 || ref >= q.nstreams) return "operand is neither a stream of the field nor a register";
    if (q.stream[ref].role == BR_OUT) return "operand stream is an output of this launch";
    kind = q.stream[ref].kind;
    return nullptr;
  };
  for (int k = 0; k < q.nsteps; k++) {
    const qlagpu_batch_step& s = q.step[k];
    BStep& d = b.st[k];
    int kind_b = -1;
    d.eqop = s.eqop;
    d.mu = s.mu;
    d.sign = s.sign == 1 ? 1 : -1;
    d.r = s.r;
    load_stream[k] = -1;
    if (s.op < 0 || s.op > 4) return plan_error(who, f, k, "unknown op");
    if (s.eqop < 0 || s.eqop > 3) return plan_error(who, f, k, "eqop out of range");
    if (s.dst != kReg0 && s.dst != kReg1) return plan_error(who, f, k, "dst must be QLAGPU_REG0 or QLAGPU_REG1");
    if (const char* e = opnd_kind(s.a, kind_a[k])) return plan_error(who, f, k, e);
    switch (s.op) {
      case BOP_LMULT:
        if (kind_a[k] != BK_M) return plan_error(who, f, k, "LMULT: a must be a colour matrix");
        if (const char* e = opnd_kind(s.b, kind_b)) return plan_error(who, f, k, e);
        if (s.adjb && kind_b != BK_M) return plan_error(who, f, k, "LMULT: adjb needs a colour-matrix b");
        kind_r[k] = kind_b;
        d.code = SC_LMULT + kind_b * 4 + (s.adja ? 2 : 0) + (s.adjb ? 1 : 0);
        break;
      case BOP_SPPROJ:
        if (kind_a[k] != BK_D) return plan_error(who, f, k, "SPPROJ: a must be a DiracFermion");
        if (s.mu < 0 || s.mu > 4) return plan_error(who, f, k, "mu must be 0..4");
        kind_r[k] = BK_H;
        d.code = SC_SPPROJ;
        break;
      case BOP_SPRECON:
        if (kind_a[k] != BK_H) return plan_error(who, f, k, "SPRECON: a must be a HalfFermion");
        if (s.mu < 0 || s.mu > 4) return plan_error(who, f, k, "mu must be 0..4");
        kind_r[k] = BK_D;
        d.code = SC_SPRECON;
        break;
      default:
        kind_r[k] = kind_a[k];
        d.code = (s.op == BOP_RTIMES ? SC_RTIMES : SC_COPY) + kind_r[k];
        break;
    }
    if (s.store >= 0) {
      if (s.store >= q.nstreams || q.stream[s.store].role == BR_IN)
        return plan_error(who, f, k, "store must name an OUT or INOUT stream");
      if (q.stream[s.store].kind != kind_r[k]) return plan_error(who, f, k, "stored stream has another kind");
      if (store_step[s.store] >= 0) return plan_error(who, f, k, "a stream is stored by more than one step");
      store_step[s.store] = k;
    } else if (s.store != -1) {
      return plan_error(who, f, k, "store must be a stream or -1");
    }
    if (s.eqop == PEQ || s.eqop == MEQ) {
      if (s.store >= 0 && q.stream[s.store].role == BR_INOUT) {
        load_stream[k] = s.store;
      } else if (regkind[s.dst - kReg0] != kind_r[k]) {
        return plan_error(who, f, k, "peq / meq needs an INOUT store stream or a dst register of the result kind");
      }
    }
    regkind[s.dst - kReg0] = kind_r[k];
  }
  for (int j = 0; j < q.nstreams; j++)
    if (q.stream[j].role != BR_IN && store_step[j] < 0)
      return plan_error(who, f, -1, "an output stream is never stored");

  // last step that reads each stream (-1: none)
  int last_read[kMaxStreams];
  for (int j = 0; j < kMaxStreams; j++) last_read[j] = -1;
  for (int k = 0; k < q.nsteps; k++) {
    const qlagpu_batch_step& s = q.step[k];
    if (s.a < kMaxStreams) last_read[s.a] = k;
    if (s.op == BOP_LMULT && s.b < kMaxStreams) last_read[s.b] = k;
    if (load_stream[k] >= 0) last_read[load_stream[k]] = k;
  }
  // Places.  Every value a step reads or makes has a region of the stage: the
  // streams' records from the start, a result from its step on.  A result
  // takes the smallest region that fits of those whose value has been read
  // for the last time (by this step at the latest), else a new one.  Values
  // that are stored stay until the tile's end.
  struct Region {
    unsigned off, size;
    int until;  // last step that reads its value; nsteps: stored at the end
  };
  std::vector<Region> regions;
  unsigned fixed = 0, stage = 0;
  // a tile's cost, in units of a site's bytes: 200 for the loop itself, 40 per
  // step, a byte per byte, a half per floating-point operation (fitted to the
  // times of five programs run alone, which it gives within 10 %)
  cost = 200 + 40 * q.nsteps;
  int stream_region[kMaxStreams], reg_region[2] = {-1, -1};
  auto new_region = [&](unsigned size, int until) {
    regions.push_back(Region{stage, size, until});
    stage += size;
    return (int)regions.size() - 1;
  };
  for (int j = 0; j < q.nstreams; j++) {
    BStream& d = b.s[j];
    stream_region[j] = -1;
    d.used = last_read[j] >= 0;
    if (d.used) {
      stream_region[j] = new_region(32u * rec_b(d.kind), last_read[j]);
      d.slot = regions[(size_t)stream_region[j]].off;
      cost += rec_b(d.kind) + (d.idx ? 4u : 0u);
      if (!d.idx) {
        b.tx += 32u * rec_b(d.kind);
        if (!d.wide) b.bulk = 0;
      } else {
        d.idx_slot = fixed;
        fixed += 3u * 128u;
        b.gather[b.ngather++] = j;
      }
    }
    if (d.role == BR_IN) continue;
    if (!d.wide) b.bulk = 0;
    cost += rec_b(d.kind);
  }
  // steps that read step k's result through its register, the last of them
  auto last_use = [&](int k) {
    const int r = q.step[k].dst;
    int last = k;
    for (int m = k + 1; m < q.nsteps; m++) {
      const qlagpu_batch_step& s = q.step[m];
      if (s.a == r || (s.op == BOP_LMULT && s.b == r) ||
          ((s.eqop == PEQ || s.eqop == MEQ) && load_stream[m] < 0 && s.dst == r))
        last = m;
      if (s.dst == r) break;
    }
    return last;
  };
  for (int k = 0; k < q.nsteps; k++) {
    const qlagpu_batch_step& s = q.step[k];
    BStep& d = b.st[k];
    const int dr = s.dst - kReg0;
    auto region_of = [&](int ref) { return ref >= kReg0 ? reg_region[ref - kReg0] : stream_region[ref]; };
    d.a = regions[(size_t)region_of(s.a)].off;
    if (s.op == BOP_LMULT) d.b = regions[(size_t)region_of(s.b)].off;
    if (s.eqop == PEQ || s.eqop == MEQ)
      d.old = regions[(size_t)(load_stream[k] >= 0 ? stream_region[load_stream[k]] : reg_region[dr])].off;
    const unsigned need = 32u * rec_b(kind_r[k]);
    int best = -1;
    for (int m = 0; m < (int)regions.size(); m++)
      if (regions[(size_t)m].until <= k && regions[(size_t)m].size >= need &&
          (best < 0 || regions[(size_t)m].size < regions[(size_t)best].size))
        best = m;
    if (best < 0) best = new_region(need, 0);
    regions[(size_t)best].until = s.store >= 0 ? q.nsteps : last_use(k);
    d.res = regions[(size_t)best].off;
    if (s.store >= 0) b.s[s.store].out = d.res;
    reg_region[dr] = best;
    cost += (s.op == BOP_LMULT ? 24 : 2) * kncplx(kind_r[k]) / 2;
  }
  if (fixed > fixed_bytes) fixed_bytes = fixed;
  if (stage > stage_bytes) stage_bytes = stage;
  return true;
}

static BatchPlan* make_plan(const char* who, const qlagpu_F3_batch_program* fields, int nfields) {
  if (!fields || nfields <= 0 || nfields > kMaxFields) {
    set_error(QLAGPU_ERR_ARG, who, "need 1 <= nfields <= 1024 and a field table");
    return nullptr;
  }
  int t = 128, st = 0;  // threads per block (the table's stages do not apply here)
  if (!tuned_shape("F3_batch_program", &t, &st) || (t != 64 && t != 128)) t = 128;
  std::vector<BField> h((size_t)nfields);
  std::vector<long long> cost((size_t)nfields);  // of a tile
  unsigned fixed_bytes = 0, stage_bytes = 0;
  long long tiles = 0;
  double total = 0.0;
  for (int f = 0; f < nfields; f++) {
    if (!build_field(who, f, fields[f], h[(size_t)f], fixed_bytes, stage_bytes, cost[(size_t)f])) return nullptr;
    h[(size_t)f].tile0 = tiles;
    const long long ft = (fields[f].n + 31) / 32;
    tiles += ft;
    total += (double)ft * (double)cost[(size_t)f];
  }
  if (!device_error_word()) return nullptr;  // allocate it now, not inside a later capture
  BatchPlan* plan = new BatchPlan();
  plan->nfields = nfields;
  plan->ntiles = tiles;
  plan->fixed_bytes = fixed_bytes;
  plan->stage_bytes = stage_bytes;
  // Two stages hide a tile's copies behind the one before it; one stage leaves
  // room for more warps, up to the 16 that the registers allow on an SM.  Two
  // where they still leave 16.  Measured on B200, two stages / one: 64 fields
  // of config 4's pair 500 us (16 warps) / 576 us (16); 30 fields of a Wilson
  // hop direction 205 (12) / 191 (16); five programs in one plan 356 (12) / 327
  // (16).
  const void* fn = reinterpret_cast<const void*>(&batch_program_kernel);
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  int nb = 1;
  for (plan->stages = 2;; plan->stages = 1) {
    plan->warp_bytes =
        (16u + 16u * (unsigned)kDescWords + fixed_bytes + (unsigned)plan->stages * stage_bytes + 127u) & ~127u;
    plan->smem = (size_t)(t / 32) * plan->warp_bytes;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, t, plan->smem) != cudaSuccess) nb = 0;
    cudaGetLastError();
    if (plan->stages == 1 || nb * (t / 32) >= 16) break;
  }
  // very large programs: narrower blocks until one fits
  while (nb < 1 && t > 32) {
    t /= 2;
    plan->smem = (size_t)(t / 32) * plan->warp_bytes;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, t, plan->smem) != cudaSuccess) nb = 0;
    cudaGetLastError();
  }
  if (nb < 1) nb = 1;
  plan->threads = t;
  const int nw = t / 32;
  long long grid = (long long)nb * device_sm_count();
  if (grid * nw > tiles) grid = (tiles + nw - 1) / nw;
  plan->grid = (int)(grid < 1 ? 1 : grid);
  // The tiles go to the blocks in contiguous runs of equal estimated cost.
  // Fields with one program: one run per block (its first tile pays the
  // index and record latencies once).  Different programs: two runs each, of
  // different parts of the list, which evens out what the cost model gets
  // wrong.  Measured, runs per block 1 / 2 / 4: five programs in one plan 326 /
  // 314 / 328 us, 64 fields of config 4's pair 507 / 510 / 506, 30 fields of a
  // hop direction 189 / 197 / 202.
  bool same = true;
  for (int f = 1; f < nfields; f++) {
    const BField &x = h[0], &y = h[(size_t)f];
    same = same && x.nsteps == y.nsteps;
    for (int k = 0; same && k < x.nsteps; k++) same = x.st[k].code == y.st[k].code;
  }
  const long long runs = (long long)plan->grid * (same || tiles < 16LL * plan->grid * nw ? 1 : 2);
  plan->runs = (int)runs;
  std::vector<long long> start((size_t)runs + 1);
  {
    int f = 0;
    double before = 0.0;  // cost of the fields before f
    for (long long w = 0; w < runs; w++) {
      const double want = total * (double)w / (double)runs;
      while (f + 1 < nfields) {
        const double here = (double)((h[(size_t)f].n + 31) / 32) * (double)cost[(size_t)f];
        if (before + here > want) break;
        before += here;
        f++;
      }
      const double c = (double)(cost[(size_t)f] > 0 ? cost[(size_t)f] : 1);
      long long g = h[(size_t)f].tile0 + (long long)((want - before) / c);
      if (g > tiles) g = tiles;
      if (w > 0 && g < start[(size_t)w - 1]) g = start[(size_t)w - 1];
      start[(size_t)w] = g;
    }
    start[0] = 0;
    start[(size_t)runs] = tiles;
  }
  const size_t fb = sizeof(BField) * (size_t)nfields, sb = sizeof(long long) * start.size();
  char* table = nullptr;
  if (cudaMalloc(&table, fb + sb) != cudaSuccess ||
      cudaMemcpy(table, h.data(), fb, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(table + fb, start.data(), sb, cudaMemcpyHostToDevice) != cudaSuccess) {
    check_launch(who);
    set_error(QLAGPU_ERR_ALLOC, who, "plan table allocation failed");
    cudaFree(table);
    delete plan;
    return nullptr;
  }
  plan->dfields = reinterpret_cast<BField*>(table);
  plan->dstart = reinterpret_cast<long long*>(table + fb);
  return plan;
}

}  // namespace qlab

using namespace qlab;

extern "C" QLAB_EXPORT void* qlagpu_F3_batch_plan_program(const qlagpu_F3_batch_program* fields, int nfields) {
  return make_plan("qlagpu_F3_batch_plan_program", fields, nfields);
}

// The fixed sequence r = u * u2[nbr] (QLA_F3_M_eq_M_times_xM), w = r * v
// (QLA_F3_V_veq_M_times_V) as a two-step program per field.
extern "C" QLAB_EXPORT void* qlagpu_F3_batch_plan(const qlagpu_F3_batch_field* fields, int nfields) {
  const char* who = "qlagpu_F3_batch_plan";
  if (!fields || nfields <= 0 || nfields > kMaxFields) {
    set_error(QLAGPU_ERR_ARG, who, "need 1 <= nfields <= 1024 and a field table");
    return nullptr;
  }
  std::vector<qlagpu_F3_batch_program> prog((size_t)nfields);
  for (int f = 0; f < nfields; f++) {
    const qlagpu_F3_batch_field& q = fields[f];
    if (!q.r || !q.u || !q.u2 || !q.nbr || !q.w || !q.v || q.n < 0) {
      set_error(QLAGPU_ERR_NULLPTR, who, "NULL array in a field (or n < 0)");
      return nullptr;
    }
    qlagpu_F3_batch_program& p = prog[(size_t)f];
    std::memset(&p, 0, sizeof(p));
    p.n = q.n;
    p.nstreams = 5;
    p.nsteps = 2;
    p.stream[0] = qlagpu_batch_stream{q.u, nullptr, 0, QLAGPU_REC_M, QLAGPU_STREAM_IN};
    p.stream[1] = qlagpu_batch_stream{q.u2, q.nbr, 0, QLAGPU_REC_M, QLAGPU_STREAM_IN};
    p.stream[2] = qlagpu_batch_stream{q.v, nullptr, 0, QLAGPU_REC_V, QLAGPU_STREAM_IN};
    p.stream[3] = qlagpu_batch_stream{q.r, nullptr, 0, QLAGPU_REC_M, QLAGPU_STREAM_OUT};
    p.stream[4] = qlagpu_batch_stream{q.w, nullptr, 0, QLAGPU_REC_V, QLAGPU_STREAM_OUT};
    p.step[0] = qlagpu_batch_step{QLAGPU_BOP_LMULT, QLAGPU_EQ, 0, 1, QLAGPU_REG0, 3, 0, 0, 0, 1, 0.f};
    p.step[1] = qlagpu_batch_step{QLAGPU_BOP_LMULT, QLAGPU_EQ, QLAGPU_REG0, 2, QLAGPU_REG1, 4, 0, 0, 0, 1, 0.f};
  }
  return make_plan(who, prog.data(), nfields);
}

extern "C" QLAB_EXPORT int qlagpu_batch_run(void* handle) {
  QLAB_TRACE("qlagpu_batch_run");
  BatchPlan* plan = static_cast<BatchPlan*>(handle);
  if (!plan) {
    set_error(QLAGPU_ERR_NULLPTR, "qlagpu_batch_run", "NULL plan");
    return QLAGPU_ERR_NULLPTR;
  }
  if (plan->ntiles == 0) return QLAGPU_OK;
  BatchParams p;
  p.fields = plan->dfields;
  p.start = plan->dstart;
  p.nfields = plan->nfields;
  p.fixed_bytes = plan->fixed_bytes;
  p.stage_bytes = plan->stage_bytes;
  p.warp_bytes = plan->warp_bytes;
  p.stages = plan->stages;
  p.runs = plan->runs;
  p.err = device_error_word();
  if (launch_kernel(&batch_program_kernel, (unsigned)plan->grid, (unsigned)plan->threads, plan->smem, current_stream(),
                    p) != cudaSuccess) {
    check_launch("qlagpu_batch_run");
    return QLAGPU_ERR_LAUNCH;
  }
  return check_launch("qlagpu_batch_run") ? QLAGPU_OK : QLAGPU_ERR_LAUNCH;
}

extern "C" QLAB_EXPORT void qlagpu_batch_destroy(void* handle) {
  BatchPlan* plan = static_cast<BatchPlan*>(handle);
  if (!plan) return;
  cudaFree(plan->dfields);
  delete plan;
}
