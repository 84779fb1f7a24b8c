// saom_common.cuh -- device-side problem descriptor and small helpers of the
// GB300 SAOM period simulator.
#pragma once
#ifdef __CUDACC_RTC__
// compiled at run time by NVRTC (saom_jit.cu): device code only, no host headers
typedef unsigned int uint32_t;
typedef int int32_t;
typedef unsigned long long uint64_t;
typedef long long int64_t;
typedef unsigned char uint8_t;
typedef unsigned short uint16_t;
typedef unsigned long long uintptr_t;
#define INFINITY __int_as_float(0x7f800000)
#else
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>
#endif

namespace cusna {

// Runaway-chain cap of the CPU engine (src/libcusna_saom_cpu.cpp:115).
constexpr long long kMaxSteps = 4000000;
constexpr int kMaxEff = 24;  // network effects per model (CUSNA_MAXEFF)
constexpr unsigned kFull = 0xFFFFFFFFu;

// Problem flags (DevProblem::flags).
enum : int {
  F_NEED_TP = 1 << 0,      // transTies: masks of the h with 0 / 1 two-paths i -> h
  F_NEED_RDEG = 1 << 1,    // reciAct: reciprocated degree of i
  F_NEED_GW29 = 1 << 2,    // gwdspFF: per-h weight differences over tp
  F_NEED_GW30 = 1 << 3,    // gwdspFB: per-h weight differences over |out_i & out_h|
  F_WANT_ENDS = 1 << 4,    // dense end networks requested
  F_HAS_INTER = 1 << 5,    // interaction effects present
  F_THETA_TAB = 1 << 13,   // term tables hold theta_e * d for every chain
  F_HAS_STEP = 1 << 14,    // some effect is constant within a ministep
  F_HAS_Z = 1 << 15,       // behaviour values are read (behaviour or dynamic covariates)
  F_LSE64 = 1 << 16,       // score log-sum-exp in float64 at every ministep (validation)
  F_NO_SCORES = 1 << 17,   // no scores requested: the score sums are not formed
};

// How the change statistic d_e of toggling i -> j is formed (DevProblem::ekind).
// Every kind yields d_e = delta * magnitude, the reference's value, and with
// F_THETA_TAB the term theta_e * d_e comes from a table of theta_e * magnitude
// (theta_e * (-m) = -(theta_e * m) exactly, so the table needs no sign).
enum : int {
  K_GEN = 0,   // computed in full per alter (gwdsp, interactions, large dyadic)
  K_CNT = 1,   // integer magnitude c (ecfn selects which count); term table T[c]
  K_LOOK = 2,  // magnitude D[idx], term T[idx]; idx from ecfn (sqrt, gw weight,
               // alter covariate, dyadic covariate tables)
  K_STEP = 3,  // magnitude depends only on (i, a_ij, a_ji): formed per ministep
  K_ZERO = 4,  // the dyadic covariate X, which the CPU engine zero-fills
  K_CROSS = 5, // multi-network cross effect (ecfn = type 33..37) reading network eoffd
};

// Multi-network problem: what the multi-network kernel needs beyond the
// per-network problems (one DevProblem per network, holding its effects).
constexpr int kMaxNet = 4;  // CUSNA_MAXNET
struct MultiDev {
  int D, n, W, nact, k;
  const int *act;                 // nact active actors first
  const float *lam;               // M*D rates
  uint32_t k0, k1;                // Philox key
  int goff[kMaxNet + 1];          // network d's effects: gidx[goff[d] .. goff[d+1])
  const int *gidx;                // their indices in the caller's effect order
  float *rscores, *scores;        // device outputs (any may be null)
  double *ntim;
  int *steps;
  uint8_t *a_ends;
};

// Two-path counters. The change statistics of a ministep need, for every alter
// j, the number of h in some set of actors that depends on the focal actor i
// alone (its out- or in-neighbours, ...) with a tie between h and j. Counter c
// is one such set and one relation of h and j (with m2, the sum over two).
//   set:      CL_OUT out_i, CL_IN in_i, CL_MUTUAL out_i & in_i, CL_TP0 / CL_TP1
//             the h of out_i with 0 / 1 two-paths i -> h (by counter tp),
//             CL_NET + w out_i in network w
//   relation: CM_ROWS a tie h -> j, CM_COLS a tie j -> h, CM_NCOLS + w a tie
//             j -> h in network w
// Those of CL_OUT, CL_IN and CL_NET are matrix products of the networks; a chain
// may hold them (mask) as n x n matrices of counts that every toggle updates
// (saom_kernel.cuh, counts_toggle), so that the pass over the alters reads row i.
enum : int { CL_OUT = 0, CL_IN = 1, CL_MUTUAL = 2, CL_TP0 = 3, CL_TP1 = 4, CL_NET = 5 };
enum : int { CM_ROWS = 0, CM_COLS = 1, CM_NCOLS = 2, CM_NONE = 255 };
constexpr int kMaxCnt = 16, kMaxTask = 32;
// One update of a count matrix when the network's tie u -> v toggles: every
// member x of a set of u's or v's neighbours (in network set_net, its out- or
// in-neighbours) changes the cell (fix, x), or by column (x, fix), fix being u or
// v, of matrix `rank` of network `net`.
constexpr unsigned task_pack(bool set_in, bool set_of_v, bool fix_v, bool by_col, int rank,
                             int set_net, int net) {
  return (unsigned)set_in | (unsigned)set_of_v << 1 | (unsigned)fix_v << 2 |
         (unsigned)by_col << 3 | (unsigned)rank << 4 | (unsigned)set_net << 8 | (unsigned)net << 12;
}
struct CounterSet {
  int n;
  int tp, tq;     // the counter of |out_i & in_h| and |out_i & out_h|, where read by h
  unsigned mask;  // counters held as matrices
  unsigned char list[kMaxCnt], m1[kMaxCnt], m2[kMaxCnt];
  int ntask;      // updates of a toggle in this network
  unsigned task[kMaxTask];
};
// Counts per matrix: n*n padded so that every matrix starts on 16 bytes (they
// are copied 16 bytes and updated 4 bytes at a time).
__host__ __device__ constexpr size_t cm_size(int n) {
  return ((size_t)n * n + 7) & ~(size_t)7;
}
// An effect's count function packed with its counters a, b, c (0xFF: none).
constexpr int cfn_pack(int fn, int a = 0xFF, int b = 0xFF, int c = 0xFF) {
  return fn | (a << 8) | (b << 16) | (int)((unsigned)c << 24);
}

// Canonical device form of one cusna_saom_problem. Every network is stored
// word-major: element (w, j) of an n-actor bit matrix is word w of actor j's
// row, at index w*n + j. Word w of row i, bit b, is the tie i -> 32*w + b.
struct DevProblem {
  int n, W, k, kb, nrate, M;
  uint32_t chain_offset;
  int cond, target_dist, symflag, maxdeg, has_comp, nact;
  uint32_t k0, k1;
  int flags;
  int zmin, zmax;
  int zlo, zR;  // range of reachable behaviour values (lookup tables)
  double zbar, brange, bsimmean;

  // effect descriptors
  const int *type_ids, *etypes, *dyn, *int0, *int1, *int2;  // k
  const double *p1, *p2;                                    // k
  const double *vmat;                                       // k*n
  const double *wtab;                                       // k*(n+1)
  const uint8_t *vmiss;                                     // k*n or null
  const double *vb;                                         // n (statistics)
  const int *od0, *id0;                                     // n or null
  const int *bty;                                           // kb
  const int *rkind;                                         // nrate
  const double *ralpha, *ru;                                // nrate, nrate*n
  const int *act;                                           // n
  const uint32_t *inact;                                    // W bits
  const int *z0, *bkdist;                                   // n

  // networks, word-major W*n (rows and, with suffix c, in-rows)
  const uint32_t *x0r, *x0c, *simr, *simc, *kdistr, *permr;
  const uint32_t *keepr, *forcer, *keepc, *forcec;       // statistic masks

  // per-chain parameters: chain c reads row c * prow (prow 1: one row per
  // chain, as the ABI lays them out; 0: one row shared by every chain)
  const float *lam, *theta, *lamb, *thetab;
  int prow;

  // effect plan (k each) and its table pool
  const int *ekind, *ecfn, *eoffd, *eofft;
  CounterSet cnt;
  const uint16_t *c0;  // start values of the counters held as matrices, cm_size(n) each
  const double *tab;
  // tab's lookup values in fixed point (see the scales below); entries 0..255 of
  // both pools are exp_fx's table
  const uint64_t *tabq;
  const double *ebound;  // k  bound on |d_e|

  // outputs (chain-major), any may be null
  double *stats, *ntim;
  float *scores;
  int *dist, *dist_stat, *steps;
  int *bdist;
  float *bscores;
  int *z_end;
  float *rscores;
  int *actor_dist;
  uint8_t *a_ends;

  // validation mode (period_kernel<MAXT, true> only): per-ministep trace
  // records (step, actor, choice, distance change), trace_cap per chain, and
  // caller-supplied words replacing the Philox outputs of the first
  // ustream_steps ministeps of each chain (4 + n words per ministep)
  int *trace;
  int trace_cap;
  const uint32_t *ustream;
  int ustream_steps;
};

// ---- Philox4x32-10 (the generator of src/libcusna_saom_cpu.cpp:32-45) ----
__host__ __device__ __forceinline__ void philox10(uint32_t c0, uint32_t c1, uint32_t c2,
                                                  uint32_t c3, uint32_t k0, uint32_t k1,
                                                  uint32_t out[4]) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
#ifdef __CUDA_ARCH__
    uint32_t hi0 = __umulhi(0xD2511F53u, c0), hi1 = __umulhi(0xCD9E8D57u, c2);
#else
    uint32_t hi0 = (uint32_t)(((uint64_t)0xD2511F53u * c0) >> 32);
    uint32_t hi1 = (uint32_t)(((uint64_t)0xCD9E8D57u * c2) >> 32);
#endif
    uint32_t lo0 = 0xD2511F53u * c0, lo1 = 0xCD9E8D57u * c2;
    uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// u = (x + 0.5) 2^-32, computed exactly in float64.
__device__ __forceinline__ double unif01(uint32_t x) {
  return __dmul_rn(__dadd_rn((double)x, 0.5), 2.3283064365386962890625e-10);
}

// Monotone int64 key of a double: a < b  <=>  dkey(a) < dkey(b) (no NaNs).
// Lets max/argmax over doubles run on the integer pipes.
__device__ __forceinline__ long long dkey(double x) {
  long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFLL);
}
__device__ __forceinline__ double dunkey(long long k) {
  long long b = k ^ ((k >> 63) & 0x7FFFFFFFFFFFFFFFLL);
  return __longlong_as_double(b);
}

// float32 estimate of log(-log(u)), u = (x + 0.5) 2^-32, by CUDA's logf and log1pf: the
// yardstick in float32 of gumbel_est below, which the kernels use. Error bound (from the documented <= 1 ulp error of
// logf/log1pf and the 2^-24 rounding of the inputs):
//   L = -log(u) is estimated with relative error < 5e-7 (for u >= 1/2 through
//   log1p of v = 1 - u, which is formed exactly from ~x), and log(L) lies in
//   [-22.9, 3.2], so |estimate - log(-log u)| < 5e-7 + 23 * 1.2e-7 < 4e-6.
__device__ __forceinline__ float loglog_est(uint32_t x) {
  float L;
  if (x < 0x80000000u) {
    float uf = ((float)x + 0.5f) * 2.3283064365386962890625e-10f;
    L = -logf(uf);
  } else {
    float vf = ((float)(0xFFFFFFFFu - x) + 0.5f) * 2.3283064365386962890625e-10f;
    L = -log1pf(-vf);
  }
  return logf(L);
}

// Faster estimate of log(-log u) for the Gumbel keys, 14 instructions without a
// branch (loglog_est above: about 80, both branches of every warp). With the
// documented errors of lg2.approx.f32 (2^-22 absolute on (0.5, 2), 2^-22
// relative elsewhere):
//   L = -log u: below v = 1 - u = 1/16 the series v + v^2/2 + v^3/3 + v^4/4
//   (omitted terms under v^4/5 = 3.1e-6 relative), else -ln2 lg2(u), relative
//   error under (1.7e-7 + 3e-8) / L = 3.1e-6 at L = 1/16; log L then adds
//   2^-22 ln2 |lg2 L| <= 5.5e-6 for L in [1e-10, 23]: 1e-5 in all, kGumbelErr.
constexpr float kGumbelErr = 1.5e-5f;
__device__ __forceinline__ float lg2_approx(float x) {
  float r;
  asm("lg2.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float gumbel_est(uint32_t x) {
  const float u = fmaf((float)x, 2.3283064365386962890625e-10f, 1.16415321826934814453125e-10f);
  const float v = fmaf((float)~x, 2.3283064365386962890625e-10f, 1.16415321826934814453125e-10f);
  const float a = __fmul_rn(lg2_approx(u), -0.693147180559945f);
  const float b = __fmul_rn(v, fmaf(v, fmaf(v, fmaf(v, 0.25f, 0.33333333f), 0.5f), 1.f));
  return __fmul_rn(lg2_approx(v < 0.0625f ? b : a), 0.693147180559945f);
}

// ---- fixed-point arithmetic of the pass over the alters ------------------------
// A ministep's predictors and score sums are 64-bit integers: their sums are
// exact whatever the order, so any split of the alters over warps gives the
// same bits, and a count's term is one 64-bit multiply-add.
//   predictor f_j          scale 2^-46 (kFBits)
//   weight exp(f_j)        scale 2^-(44 - sh) (kWBits): "no change" weighs 1; sh
//                          follows the ministep's largest predictor. Where the
//                          grid is too coarse for a sum, the ministep's sums are
//                          formed in float64 (net_choice)
//   real statistic d_e     |d_e| 2^sd + 2^62 as an unsigned number, sd_e from
//                          the effect's largest |d_e| (fx_scale)
constexpr int kFBits = 46, kWBits = 44;

// Largest sd with |d| 2^sd < 2^62 for every |d| <= bound (0: a bound of 1).
__host__ __device__ inline int fx_scale(double bound) {
  int p = 0;
  if (!(bound > 0.0)) bound = 1.0;
#ifdef __CUDA_ARCH__
  p = (int)((__double_as_longlong(bound) >> 52) & 0x7FF) - 1022;   // bound < 2^p
#else
  std::frexp(bound, &p);
#endif
  return 62 - p;
}

// High 64 bits of a * b without the product of the low halves (at most 3 below
// the exact ones): a predictor's terms.
__host__ __device__ __forceinline__ uint64_t mulhi_fx(uint64_t a, uint64_t b) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
  const uint32_t bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
#ifdef __CUDA_ARCH__
  return (uint64_t)ah * bh + __umulhi(ah, bl) + __umulhi(al, bh);
#else
  return (uint64_t)ah * bh + (((uint64_t)ah * bl) >> 32) + (((uint64_t)al * bh) >> 32);
#endif
}

// a * b 2^-64, rounded to nearest: the score sums add a product per alter, and a
// cut to one side would add up over the alters and ministeps.
__host__ __device__ __forceinline__ uint64_t mulround_fx(uint64_t a, uint64_t b) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
  const uint32_t bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  const uint64_t p = (uint64_t)ah * bl + (((uint64_t)al * bl) >> 32);
  const uint64_t q = (uint64_t)al * bh + (uint32_t)p;
  return (uint64_t)ah * bh + (p >> 32) + (q >> 32) + ((uint32_t)q >> 31);
}

// -2^62: taken off a magnitude by an addition.
constexpr uint64_t kMinus62 = 3ull << 62;

// x, or -x for neg = 1. Written with the bits' complement: the negation 0 - (a - b)
// of a difference inside a chain of additions loses a borrow in code compiled for
// sm_103a (nvcc 13.0) when low words are 0 (27,296 of 65,536 sums wrong, in unsigned
// arithmetic throughout, so no undefined behaviour enters; a - b and b - a in its
// place, or this form, 0 wrong). The fixed-point code therefore negates here only,
// and its sums, which may wrap on the way, are unsigned.
__host__ __device__ __forceinline__ int64_t signed_fx(uint64_t x, int neg) {
  const uint32_t s = 0u - (uint32_t)neg;
  return (int64_t)((x ^ ((uint64_t)s << 32 | s)) + (uint32_t)neg);
}

// exp(f 2^-46) 2^(44 - sh) rounded, for |f| < 2^61 and a result below 2^63, by
// Tang's table-driven method (P. T. P. Tang, "Table-driven implementation of the
// exponential function in IEEE floating-point arithmetic", ACM TOMS 15(2), 1989)
// in integers: f = N ln2/256 + r with |r| <= 0.53 ln2/256 = 0.00143 at scale
// 2^-62; e^r - 1 = r + r^2/2 (from r at 2^-40: error 1.3e-15) + r^3/6 + r^4/24
// (float32; the omitted r^5/120 is 5e-17); tab[N & 255] = 2^((N & 255)/256) at
// 2^-62, as (high, signed low) words; then the power of two. Relative error
// below 3e-15 + the rounding to 2^-(44-sh).
__host__ __device__ __forceinline__ uint64_t exp_fx(int64_t f, int sh, const int2 *tab) {
  const int fh = (int)(f >> 32);   // scale 2^-14
  // N = round(f 256/ln2): 256/ln2 = 369.3299304675746 at 2^-20
  const int N = (int)(((int64_t)fh * 387270501 + ((int64_t)1 << 33)) >> 34);
  // ln2/256 at 2^-62
  const int64_t r =
      (int64_t)(((uint64_t)f << 16) + (uint64_t)(int64_t)N * (uint64_t)-12486629536330718LL);
  const int s = (int)(r >> 22);    // scale 2^-40
  const float rf = (float)s * 9.094947017729282e-13f;
  const int c3 = (int)(rf * rf * rf * (rf * 0.041666668f + 0.16666667f) * 1.152921504606847e18f);
  const int64_t e = r + (((int64_t)s * s) >> 19) + (int64_t)c3 * 4;   // c3 at 2^-60
  const int2 t = tab[N & 255];
  const int64_t T = (int64_t)((uint64_t)(uint32_t)t.x << 32) + t.y;
  const int eh = (int)(e >> 32);
  const uint32_t el = (uint32_t)e;
  const int64_t lowp = (int64_t)t.x * el + (int64_t)t.y * eh;
  const uint64_t m = (uint64_t)(T + (int64_t)t.x * eh * 4 + (lowp >> 30));
  int k = 17 - (N >> 8) + sh;      // one less than the shift, for the rounding
  if (k > 62) return 0;
  if (k < 0) k = 0;                // out of range: the caller repeats with a larger sh
  return ((m >> k) + 1) >> 1;
}

// 2^(j/256) at scale 2^-62 as exp_fx's table entry.
__host__ __device__ __forceinline__ int2 exp_fx_entry(double v) {   // v = 2^(j/256)
  const int64_t T = (int64_t)(v * 4611686018427387904.0);
  const int lo = (int)(uint32_t)T;
  int2 t;
  t.x = (int)((T - lo) >> 32);
  t.y = lo;
  return t;
}

// Bound on |d_e| of effect type t for the fixed-point scale and range check
// (vmax, wmax: the largest |covariate| and |weight|; dmax: of a table).
__host__ __device__ inline double effect_bound(int t, int n, double vmax, double wmax, double p1,
                                               double p2) {
  const double N = n, a1 = p1 < 0 ? -p1 : p1, a2 = p2 < 0 ? -p2 : p2;
  switch (t) {
    case 0: case 1: case 13: case 20: case 31: case 33: case 34: case 35: return 1.0;
    case 2: case 6: case 16: case 19: return 2.0 * N + 1.0;
    case 3: case 23: case 4: case 5: case 8: case 14: case 36: case 37: return N + 1.0;
    case 7: case 9: case 15: return N + 1.0;
    case 17: return 2.0 * N + 2.0;    // 1.5 sqrt(n + 1) at most
    case 18: return 1.0;              // min(d +- 1, p) - min(d, p)
    case 10: case 11: return vmax;
    case 12: return 1.0 + 2.0 * vmax * a1 + a2;
    case 21: return vmax * vmax;
    case 25: return 2.0 * vmax;
    case 24: case 26: case 27: case 28: return wmax;
    case 29: case 30: return 2.0 * N * wmax;
    default: return 1.0;
  }
}

}  // namespace cusna
