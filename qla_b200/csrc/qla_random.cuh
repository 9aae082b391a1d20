// qla_random.cuh -- QLA's per-site random-number generator on the device:
// uniform fills (R_*_random_S), gaussian fills of every field type
// (X_*_gaussian_S), seeding from an integer field (S_*_seed_i_I) and copies /
// masked copies of the state fields (S_*_S, S_*_S_mask_I).
//
// The generator is the reference's (lib/random/QLA_random.c:18-36): an
// exclusive-or of a 24-bit feedback shift register over seven words and a
// 32-bit congruential generator with a per-site multiplier, scaled by 2^-24.
// All of it is integer arithmetic and one exact float product, so uniform
// deviates and the states left behind are bit-identical to the reference.
// Gaussian deviates follow lib/random/QLA_gaussian.c:19-55: Box-Muller in
// double (default) or MILC's polar method (QLA_use_milc_gaussian != 0, the
// spare deviate kept in the state's addend / scale words), rounded to float.
// The polar method's double log and sqrt are CUDA's; Box-Muller's log, sqrt and
// cos are written out below for the arguments that a 24-bit deviate gives.  A
// difference of a few units in the last place of the double from the host libm
// changes the float result only where the double lies that near the midpoint of
// two floats (tests/test_gpu_box_muller.py: every radius, every angle).
//
// Fills give each thread one site (the state is sequential within a site) and
// generate the record's values in the reference's order: for each complex
// element the real part, then the imaginary part.  Seeding follows
// lib/random/QLA_seed_random.c:13-36.
#pragma once
#include "qla_ewise.cuh"

extern "C" int QLA_use_milc_gaussian;

namespace qlab {

inline int rng_milc_flag() { return QLA_use_milc_gaussian != 0 ? 1 : 0; }

struct RandState {
  unsigned r0, r1, r2, r3, r4, r5, r6, multiplier, addend, ic_state;
  float scale;
};
static_assert(sizeof(RandState) == 44, "QLA_RandomState layout");

// QLA_random's 24-bit integer: the deviate is it times 2^-24
__host__ __device__ __forceinline__ unsigned rng_bits(RandState& s) {
  const unsigned t = (((s.r5 >> 7) | (s.r6 << 17)) ^ ((s.r4 >> 1) | (s.r5 << 23))) & 0xffffffu;
  s.r6 = s.r5;
  s.r5 = s.r4;
  s.r4 = s.r3;
  s.r3 = s.r2;
  s.r2 = s.r1;
  s.r1 = s.r0;
  s.r0 = t;
  const unsigned c = s.ic_state * s.multiplier + 12345u;
  s.ic_state = c;
  // (c >> 8) & 0xffffff keeps bits 8..31 whatever the shift fills in
  return t ^ ((c >> 8) & 0xffffffu);
}
// QLA_random: uniform on [0, 1)
__host__ __device__ __forceinline__ float rng_uniform(RandState& s) {
  return (1.0f / (float)0x1000000) * (float)(int)rng_bits(s);
}

// QLA_seed_random(s, seed, index)
__host__ __device__ __forceinline__ void rng_seed(RandState& s, int seed, int index) {
  const unsigned m = 69607u + 8u * (unsigned)index;
  unsigned x = (unsigned)seed;
  unsigned w[8];
  for (int j = 0; j < 8; j++) {
    x = m * x + 12345u;
    w[j] = x;
  }
  s.r0 = (w[0] >> 8) & 0xffffffu;
  s.r1 = (w[1] >> 8) & 0xffffffu;
  s.r2 = (w[2] >> 8) & 0xffffffu;
  s.r3 = (w[3] >> 8) & 0xffffffu;
  s.r4 = (w[4] >> 8) & 0xffffffu;
  s.r5 = (w[5] >> 8) & 0xffffffu;
  s.r6 = (w[6] >> 8) & 0xffffffu;
  s.ic_state = w[7];
  s.multiplier = 100005u + 8u * (unsigned)index;
  s.addend = 12345u;
  s.scale = (float)(1.0 / (double)(float)0x1000000);
}

// the polar method's rejection loop ends with probability pi/4 per pass; the
// device form gives up (and reports it) after this many passes
constexpr int kPolarMaxPasses = 4096;

// --- Box-Muller's functions for deviates k 2^-24, 0 <= k < 2^24, in FP64
//
// log: k 2^-24 = 2^E m with m in [0.707, 1.414) after moving the upper part of
// [1, 2) down an octave; the leading seven bits of m choose c near 1/m (a
// multiple of 2^-8, so m c is exact) and log m = -log c + log1p(m c - 1), with
// |m c - 1| < 2^-7 and a polynomial of degree seven (Tang's table method, ACM
// TOMS 16 (1990); the polynomial interpolates at Chebyshev nodes, error below
// 1e-17).  c = 1 next to m = 1 on both sides, so that log of a deviate near 1
// keeps its relative accuracy.
struct alignas(16) LogEntry {
  double c, t;  // c and -log c
};
constexpr int kRngTable = 128 + 6;  // entries, with the six rows of cosine's coefficients behind them
__device__ const LogEntry kLogTable[kRngTable] = {
    {1.0, 0.0},
    {0.98828125, 0.01178795575204224},
    {0.98046875, 0.01972450534777859},
    {0.97265625, 0.027724548014854862},
    {0.96484375, 0.03578910785158528},
    {0.95703125, 0.04391923393483549},
    {0.953125, 0.048009219186360606},
    {0.9453125, 0.05623971832287608},
    {0.9375, 0.06453852113757118},
    {0.9296875, 0.07290677080808779},
    {0.92578125, 0.07711730334443129},
    {0.91796875, 0.08559193033540351},
    {0.91015625, 0.09413899091386191},
    {0.90625, 0.09844007281325252},
    {0.8984375, 0.1070981355563671},
    {0.890625, 0.1158318155251217},
    {0.88671875, 0.1202274269981598},
    {0.87890625, 0.12907704227514236},
    {0.875, 0.13353139262452263},
    {0.8671875, 0.14250006260728304},
    {0.86328125, 0.14701474296180966},
    {0.85546875, 0.15610571466306167},
    {0.8515625, 0.16068238169047347},
    {0.84375, 0.16989903679539747},
    {0.83984375, 0.17453941635189968},
    {0.83203125, 0.18388527877013736},
    {0.828125, 0.18859116980755003},
    {0.82421875, 0.19331931100349597},
    {0.81640625, 0.20284319251475147},
    {0.8125, 0.2076393647782445},
    {0.80859375, 0.2124586512141934},
    {0.80078125, 0.2221674653411543},
    {0.796875, 0.22705745063534608},
    {0.79296875, 0.23197146543777514},
    {0.7890625, 0.2369097470783577},
    {0.78125, 0.24686007793152578},
    {0.77734375, 0.2518726197550701},
    {0.7734375, 0.2569104137850272},
    {0.76953125, 0.26197371574157396},
    {0.765625, 0.26706278524904525},
    {0.7578125, 0.27731928541623435},
    {0.75390625, 0.2824872555746769},
    {0.75, 0.2876820724517809},
    {0.74609375, 0.2929040164329326},
    {0.7421875, 0.29815337231907635},
    {0.73828125, 0.3034304294199201},
    {0.734375, 0.3087354816496133},
    {0.73046875, 0.31406882762497584},
    {0.7265625, 0.3194307707663612},
    {0.72265625, 0.32482161940123766},
    {0.71875, 0.33024168687057687},
    {0.71484375, 0.33569129163814154},
    {0.7109375, 0.34117075740276714},
    {1.41015625, -0.34370051385331846},
    {1.40234375, -0.3381449440087164},
    {1.39453125, -0.3325583373000766},
    {1.38671875, -0.32694034499585334},
    {1.37890625, -0.3212906124537343},
    {1.37109375, -0.31560877898630335},
    {1.3671875, -0.3127557100038969},
    {1.359375, -0.3070250352949119},
    {1.3515625, -0.3012613305781618},
    {1.34375, -0.2954642128938359},
    {1.3359375, -0.28963329258304266},
    {1.328125, -0.2837681731306446},
    {1.32421875, -0.2808226629008878},
    {1.31640625, -0.2749054858727992},
    {1.30859375, -0.26895308734550394},
    {1.3046875, -0.26596354849713794},
    {1.296875, -0.25995752443692605},
    {1.2890625, -0.25391520998096345},
    {1.28515625, -0.25088030628580943},
    {1.27734375, -0.24478272641769092},
    {1.26953125, -0.238647737850175},
    {1.265625, -0.2355660713127669},
    {1.2578125, -0.22937410106484582},
    {1.25, -0.22314355131420976},
    {1.24609375, -0.2200136583052821},
    {1.23828125, -0.21372432939771813},
    {1.234375, -0.21056476910734964},
    {1.2265625, -0.2042155414286909},
    {1.22265625, -0.20102574606059073},
    {1.21484375, -0.19461546769967167},
    {1.2109375, -0.19139485299962947},
    {1.203125, -0.184922338494012},
    {1.19921875, -0.18167030310763468},
    {1.1953125, -0.1784076574728183},
    {1.1875, -0.17185025692665923},
    {1.18359375, -0.16855536102980667},
    {1.17578125, -0.16193282026931324},
    {1.171875, -0.15860503017663857},
    {1.16796875, -0.15526612891112396},
    {1.16015625, -0.14855469432313714},
    {1.15625, -0.1451820098444979},
    {1.15234375, -0.14179791186025734},
    {1.14453125, -0.13499516453750482},
    {1.140625, -0.13157635778871926},
    {1.13671875, -0.12814582269193003},
    {1.12890625, -0.12124924363286968},
    {1.125, -0.11778303565638346},
    {1.12109375, -0.11430477128005863},
    {1.1171875, -0.11081436634029011},
    {1.109375, -0.10379679368164356},
    {1.10546875, -0.10026945316367515},
    {1.1015625, -0.09672962645855111},
    {1.09765625, -0.0931772248541833},
    {1.08984375, -0.08603433734180316},
    {1.0859375, -0.08244366921107459},
    {1.08203125, -0.07884006170777602},
    {1.078125, -0.07522342123758753},
    {1.07421875, -0.07159365318700882},
    {1.0703125, -0.06795066190850775},
    {1.0625, -0.06062462181643484},
    {1.05859375, -0.056941376400138424},
    {1.0546875, -0.053244514518812285},
    {1.05078125, -0.04953393512227663},
    {1.046875, -0.0458095360312942},
    {1.04296875, -0.04207121392068706},
    {1.0390625, -0.0383188643021366},
    {1.03515625, -0.034552381506659735},
    {1.03125, -0.030771658666753687},
    {1.02734375, -0.026976587698202076},
    {1.0234375, -0.02316705928153438},
    {1.01953125, -0.019342962843130935},
    {1.015625, -0.015504186535965254},
    {1.01171875, -0.011650617219975274},
    {1.0078125, -0.007782140442054949},
    {1.0, 0.0},
    // cos r = 1 - r^2/2 + r^4 (...), then sin r = r + r^3 (...), highest power first
    {-1.138263220199036e-11, 2.0876146265300598e-09}, {-2.7557317271714906e-07, 2.480158729876566e-05},
    {-0.0013888888888887398, 0.041666666666666664},
    {1.5918128937554457e-10, -2.5051131840044124e-08}, {2.7557316102528646e-06, -0.00019841269836758528},
    {0.008333333333330948, -0.16666666666666666},
};
// -log(k 2^-24); table: kLogTable in shared memory.  The reference adds 1e-307
// to the deviate, which only k = 0 notices.
__device__ __forceinline__ double rng_neglog(unsigned k, const LogEntry* table) {
  if (k == 0u) return 706.89362354917204;  // -log(1e-307)
  const unsigned f = __float_as_uint((float)k);  // exact
  const unsigned j = (f >> 16) & 127u;
  const bool upper = j >= 53u;  // m > 1.414: down an octave
  const double m = __hiloint2double((int)(((f & 0x7fffffu) >> 3) + (upper ? 0x3fe00000u : 0x3ff00000u)),
                                    (int)(f << 29));
  const int E = (int)(f >> 23) - (127 + 24) + (upper ? 1 : 0);
  const double dE = __hiloint2double(0x43300000, E ^ (int)0x80000000) - 4503601774854144.0;  // E, exact
  const LogEntry e = table[j];
  const double r = fma(m, e.c, -1.0);
  double q = 0.14286871767108128;
  q = fma(q, r, -0.16667968831385005);
  q = fma(q, r, 0.19999999969856708);
  q = fma(q, r, -0.2499999996608886);
  q = fma(q, r, 0.3333333333333345);
  q = fma(q, r, -0.5000000000000013);
  const double lp = fma(r * r, q, r);
  // log 2 in two parts, the first with 40 bits: its products with E are exact
  return -(fma(dE, 0.6931471805592082, e.t) + fma(dE, 7.371002565167799e-13, lp));
}
// sqrt(x), x normal: Goldschmidt's iteration from the reciprocal square root
// approximation (about 20 bits), then one correction by the residual x - g^2
__device__ __forceinline__ double rng_sqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double g = x * y, h = 0.5 * y;
  const double e = fma(-g, h, 0.5);
  g = fma(g, e, g);
  h = fma(h, e, h);
  return fma(fma(-g, g, x), h, g);
}
// cos of the reference's angle (k 2^-23 times pi, rounded), in [0, 2 pi): minus
// the nearest multiple q of pi/2 (two parts; the first difference is exact),
// then sine or cosine of |r| <= pi/4 by one polynomial with the coefficients of
// the one or the other (Chebyshev interpolation, errors below 2e-17)
__device__ __forceinline__ double rng_cos(unsigned k, const LogEntry* table) {
  const double dk = __hiloint2double(0x43300000, (int)k) - 4503599627370496.0;  // k, exact
  const double p = __dmul_rn(dk, 3.14159265358979323846 / 8388608.0);
  const unsigned q = (k + 0x200000u) >> 22;
  const double dq = __hiloint2double(0x43300000, (int)q) - 4503599627370496.0;
  double r = fma(-dq, 1.5707963267948966, p);
  r = fma(-dq, 6.123233995736766e-17, r);
  const bool sine = q & 1u;
  const LogEntry* row = table + 128 + (sine ? 3 : 0);
  const LogEntry a = row[0], b = row[1], c = row[2];
  const double z = r * r;
  const double t = fma(fma(fma(fma(fma(a.c, z, a.t), z, b.c), z, b.t), z, c.c), z, c.t);
  const double v = sine ? fma(r * z, t, r) : fma(z, fma(z, t, -0.5), 1.0);
  return ((q + 1u) & 2u) ? -v : v;
}

// One deviate: MODE 0 QLA_random, 1 QLA_gaussian (Box-Muller), 2 QLA_gaussian
// with MILC's polar method; *bad is set when that ran out of passes
enum RngMode : int { RNG_UNIFORM = 0, RNG_GAUSS = 1, RNG_MILC = 2 };
template <int MODE>
__device__ __forceinline__ float rng_deviate(RandState& s, unsigned* bad, const LogEntry* table) {
  if constexpr (MODE == RNG_UNIFORM) {
    return rng_uniform(s);
  } else if constexpr (MODE == RNG_GAUSS) {
    const unsigned kv = rng_bits(s), kp = rng_bits(s);
    return (float)__dmul_rn(rng_sqrt(2.0 * rng_neglog(kv, table)), rng_cos(kp, table));
  } else {
    if (s.addend != 0u) {
      s.addend = 0u;
      double v1 = 0.0, v2 = 0.0, rsq = 0.0;
      int pass = 0;
      do {
        v1 = (double)rng_uniform(s);
        v2 = (double)rng_uniform(s);
        v1 = __dsub_rn(__dmul_rn(2.0, v1), 1.0);
        v2 = __dsub_rn(__dmul_rn(2.0, v2), 1.0);
        rsq = __dadd_rn(__dmul_rn(v1, v1), __dmul_rn(v2, v2));
      } while ((rsq >= 1.0 || rsq == 0.0) && ++pass < kPolarMaxPasses);
      if (pass >= kPolarMaxPasses) *bad = 1u;
      const double fac = __dsqrt_rn(__ddiv_rn(__dmul_rn(-2.0, log(rsq)), rsq));
      s.scale = (float)__dmul_rn(v1, fac);
      return (float)__dmul_rn(v2, fac);
    }
    s.addend = 1u;
    return s.scale;
  }
}

__device__ __forceinline__ RandState rng_load(const void* p) {
  const unsigned* w = static_cast<const unsigned*>(p);
  RandState s;
  s.r0 = w[0];
  s.r1 = w[1];
  s.r2 = w[2];
  s.r3 = w[3];
  s.r4 = w[4];
  s.r5 = w[5];
  s.r6 = w[6];
  s.multiplier = w[7];
  s.addend = w[8];
  s.ic_state = w[9];
  s.scale = __uint_as_float(w[10]);
  return s;
}

__device__ __forceinline__ void rng_store(void* p, const RandState& s) {
  unsigned* w = static_cast<unsigned*>(p);
  w[0] = s.r0;
  w[1] = s.r1;
  w[2] = s.r2;
  w[3] = s.r3;
  w[4] = s.r4;
  w[5] = s.r5;
  w[6] = s.r6;
  w[7] = s.multiplier;
  w[8] = s.addend;
  w[9] = s.ic_state;
  w[10] = __float_as_uint(s.scale);
}

__device__ __forceinline__ void* state_ptr(const Opnd& o, long long k) {
  return (o.mode == OM_PTR) ? const_cast<void*>(o.ptrs[k])
                            : static_cast<void*>(static_cast<char*>(const_cast<void*>(o.base)) + k * 44);
}

struct RngParams {
  void* out;
  Opnd s;          // state field (read and written)
  Opnd m;          // QLA_Int field (mask / seeding index)
  const int* gang;
  long long n;
  int nreal;       // reals per output record (1 for a real field)
  int seed;
  unsigned* err;
};

// every thread of a block: the log table into shared memory
__device__ __forceinline__ void rng_load_table(LogEntry* table) {
  for (int j = threadIdx.x; j < kRngTable; j += blockDim.x) table[j] = kLogTable[j];
  __syncthreads();
}

// uniform / gaussian fill of a field of R records (nreal reals each) whose
// states are scattered (gang index, pointers)
template <typename R, int MODE>
__global__ void __launch_bounds__(128) rng_fill_kernel(const RngParams p) {
  overlap_begin();
  __shared__ __align__(16) LogEntry table[kRngTable];
  rng_load_table(table);
  unsigned bad = 0u;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long k = p.gang ? (long long)p.gang[i] : i;
    void* sp = state_ptr(p.s, k);
    RandState s = rng_load(sp);
    R* out = static_cast<R*>(p.out) + k * p.nreal;
    for (int c = 0; c < p.nreal; c++) out[c] = (R)rng_deviate<MODE>(s, &bad, table);
    rng_store(sp, s);
  }
  if (bad) raise_dev_error(p.err, QLA_DEVERR_RNG);
}

// The same for contiguous states and records: a warp takes 32 sites.  States
// (44 B) and records pass through shared memory, so that global accesses are
// contiguous (a thread that reads and writes its own 44- and 96-B records
// touches 32 lines with every instruction), records in chunks of up to 96 B
// so that long ones (P) leave room for as many warps.  What is left is bound
// by instruction issue and the FP64 pipe; CUDA's log, cos and sqrt, which
// serve any argument, take about twice the instructions of the above.
// Measured, QLA_F3_D_veq_gaussian_S on 24^3 x 48 sites: 125 us with one
// thread per site on global memory and CUDA's functions, 87 so.
constexpr int kRngChunk = 96, kRngSlot = 112;  // bytes; the slot holds an odd number of 16-B units
constexpr int kRngWarpBytes = 1408 + 32 * kRngSlot;
template <typename R, int MODE>
__global__ void __launch_bounds__(128) rng_tile_kernel(const RngParams p) {
  overlap_begin();
  __shared__ __align__(16) LogEntry table[kRngTable];
  __shared__ __align__(16) unsigned char area[4 * kRngWarpBytes];
  rng_load_table(table);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* states = area + warp * kRngWarpBytes;
  unsigned char* slots = states + 1408;
  const long long i0 = ((long long)blockIdx.x * 4 + warp) * 32;
  if (i0 >= p.n) return;
  const int nv = p.n - i0 < 32 ? (int)(p.n - i0) : 32;
  unsigned char* gs = static_cast<unsigned char*>(const_cast<void*>(p.s.base)) + i0 * 44;
  const bool wide = nv == 32 && (reinterpret_cast<uintptr_t>(gs) & 15u) == 0;
  if (wide) {
    for (int o = lane * 16; o < 1408; o += 512) cp_async_16(states + o, gs + o);
  } else {
    for (int o = lane * 4; o < nv * 44; o += 128) cp_async_4(states + o, gs + o);
  }
  cp_async_wait_all();
  __syncwarp();
  RandState s = rng_load(states + (lane < nv ? lane : 0) * 44);
  unsigned bad = 0u;
  const int rb = p.nreal * (int)sizeof(R);  // bytes of a record: a multiple of 8, or one real
  unsigned char* out = static_cast<unsigned char*>(p.out) + i0 * rb;
  for (int done = 0; done < rb; done += kRngChunk) {
    const int cb = rb - done < kRngChunk ? rb - done : kRngChunk;
    unsigned char* mine = slots + lane * kRngSlot;
#pragma unroll 4
    for (int c = 0; c < cb; c += (int)sizeof(R))
      *reinterpret_cast<R*>(mine + c) = (R)rng_deviate<MODE>(s, &bad, table);
    __syncwarp();
    if (cb % 8 == 0) {  // 32 / (cb / 8) records at a time, an 8-B piece per lane
      const int per = cb / 8, step = 32 / per, r0 = lane / per, pc = lane - r0 * per;
      if (r0 < step)
        for (int r = r0; r < nv; r += step)
          *reinterpret_cast<uint2*>(out + r * rb + done + pc * 8) =
              *reinterpret_cast<const uint2*>(slots + r * kRngSlot + pc * 8);
    } else if (lane < nv) {  // one real per record
      *reinterpret_cast<float*>(out + lane * 4) = *reinterpret_cast<const float*>(mine);
    }
    __syncwarp();
  }
  rng_store(states + lane * 44, s);
  __syncwarp();
  if (wide) {
    for (int o = lane * 16; o < 1408; o += 512)
      *reinterpret_cast<uint4*>(gs + o) = *reinterpret_cast<const uint4*>(states + o);
  } else {
    for (int o = lane * 4; o < nv * 44; o += 128)
      *reinterpret_cast<unsigned*>(gs + o) = *reinterpret_cast<const unsigned*>(states + o);
  }
  if (bad && lane < nv) raise_dev_error(p.err, QLA_DEVERR_RNG);
}

// S_*_seed_i_I: state k = QLA_seed_random(seed, a[k])
static __global__ void __launch_bounds__(256) rng_seed_kernel(const RngParams p) {
  overlap_begin();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long k = p.gang ? (long long)p.gang[i] : i;
    const int idx = (p.m.mode == OM_PTR) ? *static_cast<const int*>(p.m.ptrs[k]) : static_cast<const int*>(p.m.base)[k];
    RandState s;
    rng_seed(s, p.seed, idx);
    rng_store(static_cast<char*>(p.out) + k * 44, s);
  }
}

// S_*_S and S_*_S_mask_I: 11 words per state, one thread per word
static __global__ void __launch_bounds__(256) rng_copy_kernel(const RngParams p, int masked) {
  overlap_begin();
  const long long total = p.n * 11;
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const long long i = g / 11;
    const int w = (int)(g - i * 11);
    const long long k = p.gang ? (long long)p.gang[i] : i;
    if (masked) {
      const int mv =
          (p.m.mode == OM_PTR) ? *static_cast<const int*>(p.m.ptrs[k]) : static_cast<const int*>(p.m.base)[k];
      if (!mv) continue;
    }
    static_cast<unsigned*>(p.out)[k * 11 + w] = static_cast<const unsigned*>(state_ptr(p.s, k))[w];
  }
}

inline bool rng_prep(const char* kid, RngParams& p, void* r, Opnd s, const int* gang, int n) {
  if (n <= 0) return false;
  if (!r || !opnd_ok(s)) {
    set_error(QLAGPU_ERR_NULLPTR, kid, "NULL argument");
    return false;
  }
  std::memset(&p, 0, sizeof(p));
  p.out = r;
  p.s = s;
  p.gang = gang;
  p.n = n;
  p.err = device_error_word();
  return true;
}

inline unsigned rng_grid(long long total, int threads) {
  const long long cap = (long long)device_sm_count() * 16;
  long long grid = (total + threads - 1) / threads;
  if (grid > cap) grid = cap;
  return (unsigned)(grid < 1 ? 1 : grid);
}

template <typename R, int MODE>
inline void rng_launch_fill(const RngParams& p) {
  // (the tile kernel writes records in 8-B pieces)
  if (p.gang == nullptr && p.s.mode == OM_CONTIG &&
      (p.nreal == 1 || (reinterpret_cast<uintptr_t>(p.out) & 7u) == 0)) {
    launch_kernel(rng_tile_kernel<R, MODE>, (unsigned)((p.n + 127) / 128), 128, 0, current_stream(), p);
    return;
  }
  // Scattered states: a thread writes its record 4 or 8 B at a time, and the lines of
  // the records in progress should stay in the L2 until they are whole.  In fields
  // larger than the L2 (126 MB; a gang index may touch twice what it counts) six blocks
  // an SM run, else sixteen.  Measured, us, sixteen / six: DN D_veq_gaussian_pS nc = 2 on
  // 750,000 sites 127 / 98, FN D_xeq_gaussian_S nc = 2 on 750,000 129 / 106, D3
  // D_xeq_gaussian_S on 694,000 278 / 243; but D3 D_xeq on 166,667 (78 MB) 39 / 43.
  unsigned grid = rng_grid(p.n, 128);
  if ((double)p.n * (p.nreal * (double)sizeof(R) + 44.0) * (p.gang ? 2.0 : 1.0) > 126e6) {
    const unsigned cap = 6u * (unsigned)device_sm_count();
    if (grid > cap) grid = cap;
  }
  launch_kernel(rng_fill_kernel<R, MODE>, grid, 128, 0, current_stream(), p);
}

// r (nreal reals per record of R) = uniform (gauss 0) or gaussian deviates
template <typename R>
inline void rng_fill(const char* kid, int nreal, int gauss, void* r, Opnd s, const int* gang, int n) {
  RngParams p;
  if (!rng_prep(kid, p, r, s, gang, n)) return;
  p.nreal = nreal;
  if (!gauss)
    rng_launch_fill<R, RNG_UNIFORM>(p);
  else if (rng_milc_flag())
    rng_launch_fill<R, RNG_MILC>(p);
  else
    rng_launch_fill<R, RNG_GAUSS>(p);
  check_launch(kid);
}

// fills of a real field (REAL) or of records of NE complex numbers
template <typename R, int NE, bool REAL>
inline void api_rng_fill(const char* kid, int gauss, void* r, Opnd s, const int* gang, int n) {
  rng_fill<R>(kid, REAL ? 1 : 2 * NE, gauss, r, s, gang, n);
}

// the same with nc colours (records of ne complex numbers)
template <typename R>
inline void api_rng_fill_n(const char* kid, int nc, int ne, int gauss, void* r, Opnd s, const int* gang, int n) {
  if (nc < 1 || nc > 64) {
    set_error(QLAGPU_ERR_ARG, kid, "nc outside 1..64");
    return;
  }
  rng_fill<R>(kid, 2 * ne, gauss, r, s, gang, n);
}

inline void api_rng_seed(const char* kid, void* r, int seed, Opnd a, const int* gang, int n) {
  RngParams p;
  if (!rng_prep(kid, p, r, Opnd{}, gang, n)) return;
  if (!opnd_ok(a)) {
    set_error(QLAGPU_ERR_NULLPTR, kid, "NULL argument");
    return;
  }
  p.m = a;
  p.seed = seed;
  launch_kernel(rng_seed_kernel, rng_grid(n, 256), 256, 0, current_stream(), p);
  check_launch(kid);
}

inline void api_rng_copy(const char* kid, void* r, Opnd a, Opnd mask, bool masked, const int* gang, int n) {
  RngParams p;
  if (!rng_prep(kid, p, r, a, gang, n)) return;
  if (masked && !opnd_ok(mask)) {
    set_error(QLAGPU_ERR_NULLPTR, kid, "NULL argument");
    return;
  }
  p.m = mask;
  launch_kernel(rng_copy_kernel, rng_grid((long long)n * 11, 256), 256, 0, current_stream(), p, masked ? 1 : 0);
  check_launch(kid);
}

}  // namespace qlab
