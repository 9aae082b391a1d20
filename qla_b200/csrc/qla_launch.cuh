// qla_launch.cuh -- host-side launch of an engine OP: path selection (bulk-copy
// pipeline or warp-cooperative kernel), tile shape, occupancy-sized persistent grid, reduction
// scratch and the synchronous host-result semantics of the reference.
#pragma once
#include <cstring>
#include <mutex>
#include <map>
#include <tuple>

#include "qla_engine.cuh"
#include "qla_runtime.h"

namespace qlab {

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

struct LaunchShape {
  int threads;  // sites per tile == threads per block
  int stages;
};

// Every kernel goes out through here, with programmatic stream serialisation:
// its blocks come onto the SMs as soon as the blocks of the kernel before have
// ended, and wait there (overlap_begin) until that kernel's writes are visible,
// so a call does not cost the stream the whole launch latency.  Order and
// results are a plain launch's; inside a captured graph the edge is a
// programmatic one.  Measured: the 24 calls of a Wilson hop on 8^4 sites 114 us
// in plain launches, 93 so; on 32^3 x 64 1472 / 1420; eight fused terms on its
// even sites 875 / 857.
template <class... P, class... A>
inline cudaError_t launch_kernel(void (*fn)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st,
                                 A&&... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fn, P(args)...);
}

// shared memory of one block of the pipelined kernel
inline size_t tma_smem_bytes(int threads, int stages, unsigned stage_bytes, unsigned out_bytes) {
  return 256 + (size_t)stages * stage_bytes + 2 * (size_t)threads * out_bytes;
}

inline unsigned stage_bytes_for(int threads, unsigned bytes_per_site) {
  return ((unsigned)threads * bytes_per_site + 127u) & ~127u;
}

// Default tile shape: two stages, and the largest tile (sites = consumer
// threads) whose block still fits in ~100 KB of shared memory, so that two to
// four blocks share an SM.  Measured on B200: more resident blocks beat deeper
// pipelines for these streaming tiles.
inline LaunchShape default_shape(unsigned bytes_per_site, unsigned out_bytes) {
  LaunchShape s{64, 2};
  for (int t : {256, 128, 64}) {
    if (tma_smem_bytes(t, 2, stage_bytes_for(t, bytes_per_site), out_bytes) <= 100u * 1024u) {
      s.threads = t;
      break;
    }
  }
  return s;
}

// resident blocks per SM of a kernel at a block shape (cached)
inline int launch_blocks_per_sm(const void* fn, int threads, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, size_t, const void*>, int> cache;
  const int dev = current_device();
  auto key = std::make_tuple(dev, threads, smem, fn);
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, threads, smem) != cudaSuccess) nb = 1;
  if (nb < 1) nb = 1;
  cache[key] = nb;
  return nb;
}

// raises a kernel's dynamic shared-memory limit to at least `smem`
inline void launch_smem_limit(const void* fn, size_t smem) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> done;
  const int dev = current_device();
  std::lock_guard<std::mutex> g(mu);
  size_t& cur = done[std::make_pair(dev, fn)];
  if (smem > cur) {
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cur = smem;
  }
}

// Lanes that meet on one bank when each reads its own record of a flat tile
// with 16-B accesses (8 lanes a phase, 4 banks each).
constexpr int bank_ways(int rec_bytes) {
  if (rec_bytes == 0 || rec_bytes % 16 != 0) return 1;  // 8-B accesses of an odd length: none
  int u = rec_bytes / 16, w = 1;
  while (w < 8 && u % 2 == 0) {
    u /= 2;
    w *= 2;
  }
  return w;
}

template <class OP>
struct SiteLauncher {
  using R = typename OP::R;
  static constexpr int RB[3] = {OP::N0 * (int)sizeof(Cx<R>), OP::N1 * (int)sizeof(Cx<R>),
                                OP::N2 * (int)sizeof(Cx<R>)};
  static constexpr int OB = OP::NOUT * (int)sizeof(Cx<R>);

  // Everything about a launch that does not depend on the arrays or n.
  struct Shape {
    // what it was made for
    const char* kernel_id = nullptr;
    int device = -1, modes = -1;
    unsigned version = 0;
    // the shape
    int threads, stages, blocks;  // blocks: resident per SM
    size_t smem;
    unsigned off_in[3], off_out_in, tx_bytes, stage_bytes;
  };

  // Warp-cooperative kernel: four warps a block, fewer where their slices would
  // leave less than four blocks an SM.  (Kept per host thread and device, like
  // tile_shape's: with the locked tables behind the tuning, the occupancy and the
  // shared-memory limit on every call, 24 short calls took 100 us, 96 so.)
  static const Shape& coop_shape() {
    static thread_local Shape sh;
    const int dev = current_device();
    if (sh.device == dev) return sh;
    constexpr unsigned wb = CoopLayout<OP>::warp_bytes;
    int nw = 4;
    while (nw > 1 && nw * wb > 48u * 1024u) nw /= 2;
    sh.threads = 32 * nw;
    sh.smem = (size_t)nw * wb;
    const void* fn = reinterpret_cast<const void*>(&site_coop_kernel<OP>);
    launch_smem_limit(fn, sh.smem);
    sh.blocks = launch_blocks_per_sm(fn, sh.threads, sh.smem);
    sh.device = dev;
    return sh;
  }

  // Bulk-copy kernel, for p's operand modes and whether the destination is
  // read: the autotuner's shape (or the default; SMALL: two stages of 64 sites)
  // and the stage layout.  Remade when the tuning table changes (tune_version).
  template <bool SMALL>
  static const Shape& tile_shape(const SiteParams& p, const char* kernel_id) {
    static thread_local Shape sh;
    const int dev = current_device();
    int modes = OP::NOUT > 0 && p.out_read ? 1 : 0;
    for (int j = 0; j < OP::NIN; j++) modes = modes * 4 + (p.in[j].mode & 3);
    const unsigned version = tune_version();
    if (sh.device == dev && sh.modes == modes && sh.version == version && sh.kernel_id == kernel_id) return sh;
    unsigned bps = 0;
    for (int j = 0; j < OP::NIN; j++)
      bps += p.in[j].mode == OM_CONTIG ? RB[j] : (p.in[j].mode == OM_PTR ? 8u : 4u);
    if (OP::NOUT > 0 && p.out_read) bps += OB;
    LaunchShape ls = default_shape(bps, OB);
    int tt, ts;
    char key[96];
    {
      int q = 0;
      for (const char* c = kernel_id; *c && q < 80; c++) key[q++] = *c;
      key[q++] = ':';
      for (int j = 0; j < OP::NIN; j++) key[q++] = "-cpi"[p.in[j].mode & 3];
      if (OP::NOUT > 0 && p.out_read) key[q++] = 'r';
      key[q] = 0;
    }
    const void* fn = reinterpret_cast<const void*>(&site_tma_kernel<OP>);
    if (SMALL) {
      ls.threads = 64;
      ls.stages = 2;
    } else if (tuned_shape(key, &tt, &ts)) {
      ls.threads = tt;
      ls.stages = ts;
    } else {
      // Where registers, not shared memory, limit the blocks on an SM, a block of
      // nine warps may leave room for much less than another one: half the
      // tile if at least a quarter more consumers fit (F3 reunit at 104
      // registers, 24^3 x 48: 8 consumer warps 49 us, 12 so 41; sqrt 110 / 98).
      auto consumers = [&](int t) {
        const size_t m = tma_smem_bytes(t, ls.stages, stage_bytes_for(t, bps), OB);
        launch_smem_limit(fn, m);
        return t * launch_blocks_per_sm(fn, t + 32, m);
      };
      while (ls.threads > 64 && 4 * consumers(ls.threads / 2) >= 5 * consumers(ls.threads)) ls.threads /= 2;
    }
    // stay within the per-block shared-memory limit (227 KB less the static
    // reduction scratch): shed stages, then halve the tile down to one warp,
    // then (very large records, e.g. nc = 8 matrices) run unpipelined
    while (tma_smem_bytes(ls.threads, ls.stages, stage_bytes_for(ls.threads, bps), OB) > 225u * 1024u) {
      if (ls.stages > 2)
        ls.stages--;
      else if (ls.threads > 32)
        ls.threads /= 2;
      else if (ls.stages > 1)
        ls.stages = 1;
      else
        break;
    }
    const int T = ls.threads;
    unsigned off = 0;
    sh.tx_bytes = 0;
    for (int j = 0; j < 3; j++) sh.off_in[j] = 0;
    for (int j = 0; j < OP::NIN; j++) {
      sh.off_in[j] = off;
      const unsigned b = (unsigned)T * (p.in[j].mode == OM_CONTIG ? RB[j] : (p.in[j].mode == OM_PTR ? 8u : 4u));
      off += (b + 15u) & ~15u;
      sh.tx_bytes += b;
    }
    sh.off_out_in = off;
    if (OP::NOUT > 0 && p.out_read) {
      off += (unsigned)T * OB;
      sh.tx_bytes += (unsigned)T * OB;
    }
    sh.stage_bytes = (off + 127u) & ~127u;
    sh.threads = T;
    sh.stages = ls.stages;
    sh.smem = tma_smem_bytes(T, sh.stages, sh.stage_bytes, OB);
    launch_smem_limit(fn, sh.smem);
    sh.blocks = launch_blocks_per_sm(fn, T + 32, sh.smem);
    sh.device = dev;
    sh.modes = modes;
    sh.version = version;
    sh.kernel_id = kernel_id;
    return sh;
  }

  // the launch has been made: its status, and a reduction's result on the host
  static void finish_call(const ReduceScratch* rs, const char* kernel_id, void* host_result, size_t result_bytes) {
    if (!check_launch(kernel_id) || OP::NACC == 0 || !host_result) return;
    cudaStream_t st = current_stream();
    if (cudaMemcpyAsync(host_result, rs->result, result_bytes, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      check_launch(kernel_id);
  }

  // Scattered calls that the warp-cooperative kernel would slow down: records so
  // short that neighbouring sites share lines, in fields that fill the GPU, and
  // operators that leave an SM three or four of its warps (FewWarps), in fields of
  // more than one round of those.  Measured on gang calls, us, warp-cooperative / one
  // site per thread: D3 norm2_V on 166,667 sites 9.6 / 6.7, F3 norm2_V on 1.39 M 15.1 /
  // 13.6, FN re_V_dot_V nc = 2 on 750,000 13.6 / 10.4, but F3 V_dot_V on 1.39 M 28 / 31
  // and FN norm2_H nc = 2 on 3.1 M 40 / 44; below 65,536 sites a few per cent the other
  // way.  FN V_xpeq_V nc = 2 on 3.1 M 60 / 50.  DN D_xpeq_M_times_D nc = 8 on 15,000 sites
  // 48 / 34, on 23,438 52 / 34, but on 1,500 29 / 34; M_xeq_M_times_M on 15,000 96 / 219.
  static bool coop_loses(const SiteParams& p, int sms) {
    constexpr int RBMAX = RB[0] > RB[1] ? (RB[0] > RB[2] ? RB[0] : RB[2]) : (RB[1] > RB[2] ? RB[1] : RB[2]);
    constexpr int SHORT = OP::NACC == 0 ? (StreamsRecords<OP>::value && OB <= 16 ? 32 : 0)
                          : sizeof(R) == 8 ? 48 : OP::NIN == 1 ? 24 : 16;
    if (RBMAX <= SHORT) return p.n > 65536;
    if (!FewWarps<OP>::value) return false;
    const Shape& sh = coop_shape();
    return p.n > (long long)sh.blocks * sh.threads * sms;
  }

  // One site per thread, in blocks of 256; of fewer threads (32 at least) while
  // blocks of twice as many would leave SMs without one (QLA_DN_M_veq_invsqrt_M,
  // nc = 8, 3,000 sites: blocks of 256 1,012 us, so 269).
  static void run_per_site(const SiteParams& p, const char* kernel_id, int sms, const ReduceScratch* rs,
                           void* host_result, size_t result_bytes) {
    int threads = 256;
    while (threads > 32 && p.n <= (long long)threads / 2 * sms) threads /= 2;
    long long grid = (p.n + threads - 1) / threads;
    if (grid > 8LL * sms) grid = 8LL * sms;
    launch_kernel(&site_direct_kernel<OP>, (unsigned)grid, (unsigned)threads, 0, current_stream(), p);
    finish_call(rs, kernel_id, host_result, result_bytes);
  }

  // kernel_id names the OP for the autotuner table
  static void run(SiteParams p, const char* kernel_id, void* host_result = nullptr, size_t result_bytes = 0) {
    constexpr bool reduce = OP::NACC > 0;
    cudaStream_t st = current_stream();
    if (p.n <= 0) {
      // the reference loops zero times; reductions still store their (zero) sum
      if (reduce) {
        if (host_result)
          std::memset(host_result, 0, result_bytes);
        else if (p.result)
          cudaMemsetAsync(p.result, 0, result_bytes, st);
      }
      return;
    }
    p.err = device_error_word();
    // ---- path selection
    bool scattered = (p.gang != nullptr);
    for (int j = 0; j < OP::NIN; j++) {
      const Opnd& o = p.in[j];
      const void* q = o.mode == OM_PTR ? (const void*)o.ptrs : (o.mode == OM_IDX ? (const void*)o.idx : o.base);
      if (!aligned16(q)) scattered = true;
    }
    if (OP::NOUT > 0 && !aligned16(p.out)) scattered = true;
    const bool per_site = scattered ? SitePerThread<OP>::scattered : SitePerThread<OP>::contiguous;
    bool direct = scattered;  // the warp-cooperative kernel
    // Records of a multiple of 128 B (4 and 8 colours' matrices and Dirac
    // fermions) lie flat in a bulk-copied tile with all eight lanes of a phase
    // on the same banks; the warp-cooperative kernel pads its slots.  Measured
    // (tile / padded slots, us): QLA_FN_M_veq_M_times_Ma nc = 4 on 320,000 sites
    // 41 / 24, nc = 8 on 41,472 sites 253 / 48; QLA_DFN_c_veq_D_dot_D nc = 4 32 /
    // 23.  Up to four ways (D3 Dirac fermions) the copies still bound the tile.
    if (bank_ways(OB) == 8) direct = true;
    for (int j = 0; j < OP::NIN; j++)
      if (p.in[j].mode == OM_CONTIG && bank_ways(RB[j]) == 8) direct = true;
    if (ComputeBound<OP>::value) direct = true;

    // ---- reduction scratch / result destination
    ReduceScratch* rs = nullptr;
    int sms = device_sm_count();
    if (reduce) {
      rs = reduce_scratch(st, 32 * sms + 64);
      if (!rs) return;
      p.partials = rs->partials;
      p.counter = rs->counter;
      if (host_result) p.result = rs->result;
    }

    if (per_site || (scattered && coop_loses(p, sms))) {
      run_per_site(p, kernel_id, sms, rs, host_result, result_bytes);
      return;
    }

    // Small fields run 64-site tiles: more SMs get a tile and the last round is
    // emptier by less.  Operators that only stream records: below three rounds
    // of the usual tiles (24 calls of a Wilson hop in a graph, usual / 64-site
    // tiles, us: 16^4 sites 90 / 87, 16^3 x 32 127 / 107, 24^4 242 / 232, but
    // 24^3 x 48 470 / 469 and 32^4 739 / 754).  Arithmetic suffers from a producer
    // warp for every two consumers (F3 sqrtPH at 65,536 sites 5.2 / 5.9, at 4,096
    // 3.9 / 3.2): while there are fewer usual tiles than SMs.  Reductions fold one
    // partial per block (F3 norm2_D at 65,536 sites 5.4 / 8.9, at 4,096 4.5 / 4.1):
    // while the 64-site tiles do not outnumber the SMs.
    const Shape* ps = direct ? &coop_shape() : &tile_shape<false>(p, kernel_id);
    if (!direct && ps->threads > 64) {
      const long long usual = (long long)ps->threads * sms;
      const long long below = reduce ? 64LL * sms : StreamsRecords<OP>::value ? 3 * usual * ps->blocks : usual;
      if (p.n < below) ps = &tile_shape<true>(p, kernel_id);
    }
    const Shape& sh = *ps;
    long long grid;
    cudaError_t rc;
    if (direct) {
      grid = (p.n + sh.threads - 1) / sh.threads;
      if (grid > (long long)sh.blocks * sms) grid = (long long)sh.blocks * sms;
      if (reduce && grid > rs->max_blocks) grid = rs->max_blocks;
      rc = launch_kernel(&site_coop_kernel<OP>, (unsigned)grid, (unsigned)sh.threads, sh.smem, st, p);
    } else {
      for (int j = 0; j < 3; j++) p.off_in[j] = sh.off_in[j];
      p.off_out_in = sh.off_out_in;
      p.tx_bytes = sh.tx_bytes;
      p.stage_bytes = sh.stage_bytes;
      p.stages = sh.stages;
      p.ntiles = p.n / sh.threads;
      grid = (long long)sh.blocks * sms;
      if (grid > p.ntiles) grid = p.ntiles;
      if (grid < 1) grid = 1;
      if (reduce && grid > rs->max_blocks) grid = rs->max_blocks;
      // threads consumers (one site each per tile) + one producer warp
      rc = launch_kernel(&site_tma_kernel<OP>, (unsigned)grid, (unsigned)sh.threads + 32u, sh.smem, st, p);
    }
    if (rc != cudaSuccess) {
      check_launch(kernel_id);
      return;
    }
    finish_call(rs, kernel_id, host_result, result_bytes);
  }
};

// operand constructors
inline Opnd op_contig(const void* base) { return Opnd{base, nullptr, nullptr, OM_CONTIG}; }
inline Opnd op_ptr(const void* const* ptrs) { return Opnd{nullptr, ptrs, nullptr, OM_PTR}; }
inline Opnd op_idx(const void* base, const int* idx) { return Opnd{base, nullptr, idx, OM_IDX}; }

inline SiteParams make_params(long long n, int eqop) {
  SiteParams p;
  std::memset(&p, 0, sizeof(p));
  p.n = n;
  p.eqop = eqop;
  p.out_read = (eqop == PEQ || eqop == MEQ) ? 1 : 0;
  return p;
}

}  // namespace qlab
