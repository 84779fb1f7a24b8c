// saom_kernel.cuh -- the GB300 period-simulator kernel.
//
// One team of G warps (G = 1, 2, 4, 8 or 16) runs one chain at a time. Teams
// take chains from a global work counter, so a launch holds one team per
// resident slot and runs until the queue is empty (a persistent kernel). Each
// team owns a slice of dynamic shared memory: the chain's out-rows and in-rows
// as word-major bitsets (or pointers to them in global scratch), degrees, behaviour values and per-alter scratch.
//
// A network ministep (src/libcusna_saom_cpu.cpp:229-287) is one pass over the
// alters j, which the team's lanes split in strides of 32*G: change statistics
// d_je from degrees and two-path counts (popcounts of the bitsets, or for larger
// networks a row of count matrices that the chain keeps up to date), the linear
// predictor f_j = sum_e theta_e d_je in 64-bit fixed point, the float32 Gumbel
// key g_j = f_j - log(-log u_j) with its error bound, and the score sums of
// exp(f_j) and exp(f_j) d_je, in fixed point as well. The keys decide the chosen
// alter when the best key's lower bound beats every other key's upper bound;
// otherwise the exact float64 keys of the alters still in range decide, ties to
// the smaller j, as the reference chooses. u_j comes from the reference's Philox
// counters (msteps, chain, 1, j), so the chosen alter, and therefore the whole
// trajectory, equals the CPU engine's.
#pragma once
#include "saom_common.cuh"

namespace cusna {

// ---------------------------------------------------------------- team sync
struct Team {
  int G, L, tl, warp, lane, bar;
  __device__ __forceinline__ void sync() const {
    if (G == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(L) : "memory");
  }
};

// Per-team shared-memory slice. Sizes depend on the launch's largest problem.
struct Slice {
  uint32_t *rows;    // W*n (shared or global scratch)
  uint32_t *cols;    // W*n (shared or global scratch)
  short *indeg, *outdeg;  // n each (degrees < 2^15 as n <= 8192)
  int *z;
  float *gbuf;       // n   upper bounds of the float32 Gumbel keys
  unsigned char *ring;  // the score sums of the last ministeps (ScoreRing), then
                     //   min(32, ceil(n/32))*(k+1) sums of the float64 path
  uint32_t *okbits;  // W
  int *tp;           // n   (gwdspFF)
  int *tq;           // n   (gwdspFB)
  uint32_t *tpeq;    // 2W  (transTies masks tp==0, tp==1)
  uint16_t *cm;      // the counters held as matrices, cm_size(n) each (global scratch)
  double *crate;     // n   (non-basic rates)
  double *red;       // 32*G + 64 reduction scratch
  int *redh;         // 32*G  high parts of the warps' score sums
  int *rfm;          // G    the warps' largest predictors (and flags)
  double *th;        // k  parameters of the current chain
  uint64_t *thq;     // k  the same in fixed point (theta_fx)
  int *esd, *ecls;   // k  scale of a real statistic, class (FX_*) of an effect
  int64_t *fx;       // 3  constant part of the predictor; in range (0/1); bound on counts
  double *sc;        // k  scores
  double *dstar;     // k  change statistics of the chosen alter
  double *thb, *bsc; // kb
  double *rsc;       // nrate
  double *p1, *p2;   // k
  int *tid, *ety, *dyn, *i0, *i1, *i2, *bty, *rkind;
  int *misc;         // 16 ints: team broadcast slots
  double *rtau;      // 32 constant-rate draws: time increments,
  int *rnet, *rfocal; //   network/behaviour flag, focal actor,
  uint32_t *rr3;     //   behaviour uniform
  int *ekind, *ecfn, *eoffd, *eofft;  // k  effect plan
  double *stepd, *stept;  // 4k  per-ministep K_STEP magnitudes and terms
  uint64_t *stepq;   // 4k  their magnitudes in fixed point
  const int2 *etab;  // exp_fx's table (the CTA's)
};

struct SliceLayout {
  size_t bytes;  // per team
  size_t o_rows, o_cols, o_indeg, o_outdeg, o_z, o_g, o_ring, o_ok, o_tp, o_tq, o_tpeq, o_crate, o_red, o_th, o_sc, o_dstar, o_thb, o_bsc, o_rsc, o_p1, o_p2, o_tid,
      o_ety, o_dyn, o_i0, o_i1, o_i2, o_bty, o_rkind, o_misc, o_rtau, o_rnet, o_rfocal, o_rr3, o_ekind, o_ecfn, o_eoffd, o_eofft,
      o_stepd, o_stept, o_stepq, o_thq, o_esd, o_ecls, o_fx, o_redh, o_rfm;
};

__host__ __device__ inline size_t al16(size_t x) { return (x + 15) & ~(size_t)15; }

// Ministeps whose score sums wait for one flush (scores_flush).
constexpr int kRing = 8;
__host__ __device__ inline size_t ring_bytes(int k) {
  return al16((size_t)kRing * ((k + 2) * 12 + k * 8 + 4));
}

// Layout of one team slice for maxima (n, k, ...) over the launch.
__host__ __device__ inline SliceLayout make_layout(int n, int W, int k, int kb, int nrate, int G,
                                                   bool rows_in_smem, bool cols_in_smem,
                                                   bool need_tp, bool need_gw, bool need_tq) {
  SliceLayout s{};
  size_t o = 0;
  auto put = [&](size_t &field, size_t bytes) { field = o; o = al16(o + bytes); };
  put(s.o_rows, rows_in_smem ? (size_t)W * n * 4 : 0);
  put(s.o_cols, cols_in_smem ? (size_t)W * n * 4 : 0);
  put(s.o_indeg, (size_t)n * 2);
  put(s.o_outdeg, (size_t)n * 2);
  put(s.o_z, (size_t)n * 4);
  put(s.o_g, (size_t)n * 4);
  put(s.o_ring, ring_bytes(k) + (size_t)(n > 992 ? 32 : (n + 31) / 32) * (k + 1) * 8);
  put(s.o_ok, (size_t)W * 4);
  put(s.o_tp, need_gw ? (size_t)n * 4 : 0);
  put(s.o_tq, need_tq ? (size_t)n * 4 : 0);
  put(s.o_tpeq, need_tp ? (size_t)W * 8 : 0);
  put(s.o_crate, nrate > 0 ? (size_t)n * 8 : 0);
  put(s.o_red, (size_t)32 * G * 8 + 64 * 8);   // 32 slots per warp, 32 results, 32 scratch
  put(s.o_th, (size_t)k * 8);
  put(s.o_sc, (size_t)k * 8);
  put(s.o_dstar, (size_t)k * 8);
  put(s.o_thb, (size_t)(kb + 1) * 8);
  put(s.o_bsc, (size_t)(kb + 1) * 8);
  put(s.o_rsc, (size_t)(nrate + 1) * 8);
  put(s.o_p1, (size_t)k * 8);
  put(s.o_p2, (size_t)k * 8);
  put(s.o_tid, (size_t)k * 4);
  put(s.o_ety, (size_t)k * 4);
  put(s.o_dyn, (size_t)k * 4);
  put(s.o_i0, (size_t)k * 4);
  put(s.o_i1, (size_t)k * 4);
  put(s.o_i2, (size_t)k * 4);
  put(s.o_bty, (size_t)(kb + 1) * 4);
  put(s.o_rkind, (size_t)(nrate + 1) * 4);
  put(s.o_misc, 16 * 4);
  put(s.o_rtau, 32 * 8);
  put(s.o_rnet, 32 * 4);
  put(s.o_rfocal, 32 * 4);
  put(s.o_rr3, 32 * 4);
  put(s.o_ekind, (size_t)k * 4);
  put(s.o_ecfn, (size_t)k * 4);
  put(s.o_eoffd, (size_t)k * 4);
  put(s.o_eofft, (size_t)k * 4);
  put(s.o_stepd, (size_t)k * 4 * 8);
  put(s.o_stept, (size_t)k * 4 * 8);
  put(s.o_stepq, (size_t)k * 4 * 8);
  put(s.o_thq, (size_t)k * 8);
  put(s.o_esd, (size_t)k * 4);
  put(s.o_ecls, (size_t)k * 4);
  put(s.o_fx, 24);
  put(s.o_redh, (size_t)32 * G * 4);
  put(s.o_rfm, (size_t)G * 4);
  s.bytes = al16(o);
  return s;
}

// A null rows or in-rows pointer: that part of the chain's state is in the slice.
__device__ __forceinline__ Slice carve(unsigned char *base, const SliceLayout &L,
                                       uint32_t *cols_global, uint32_t *rows_global,
                                       uint16_t *counts_global, const int2 *etab) {
  Slice s;
  s.rows = rows_global ? rows_global : (uint32_t *)(base + L.o_rows);
  s.cols = cols_global ? cols_global : (uint32_t *)(base + L.o_cols);
  s.indeg = (short *)(base + L.o_indeg);
  s.outdeg = (short *)(base + L.o_outdeg);
  s.z = (int *)(base + L.o_z);
  s.gbuf = (float *)(base + L.o_g);
  s.ring = base + L.o_ring;
  s.okbits = (uint32_t *)(base + L.o_ok);
  s.tp = (int *)(base + L.o_tp);
  s.tq = (int *)(base + L.o_tq);
  s.tpeq = (uint32_t *)(base + L.o_tpeq);
  s.cm = counts_global;
  s.crate = (double *)(base + L.o_crate);
  s.red = (double *)(base + L.o_red);
  s.th = (double *)(base + L.o_th);
  s.sc = (double *)(base + L.o_sc);
  s.dstar = (double *)(base + L.o_dstar);
  s.thb = (double *)(base + L.o_thb);
  s.bsc = (double *)(base + L.o_bsc);
  s.rsc = (double *)(base + L.o_rsc);
  s.p1 = (double *)(base + L.o_p1);
  s.p2 = (double *)(base + L.o_p2);
  s.tid = (int *)(base + L.o_tid);
  s.ety = (int *)(base + L.o_ety);
  s.dyn = (int *)(base + L.o_dyn);
  s.i0 = (int *)(base + L.o_i0);
  s.i1 = (int *)(base + L.o_i1);
  s.i2 = (int *)(base + L.o_i2);
  s.bty = (int *)(base + L.o_bty);
  s.rkind = (int *)(base + L.o_rkind);
  s.misc = (int *)(base + L.o_misc);
  s.rtau = (double *)(base + L.o_rtau);
  s.rnet = (int *)(base + L.o_rnet);
  s.rfocal = (int *)(base + L.o_rfocal);
  s.rr3 = (uint32_t *)(base + L.o_rr3);
  s.ekind = (int *)(base + L.o_ekind);
  s.ecfn = (int *)(base + L.o_ecfn);
  s.eoffd = (int *)(base + L.o_eoffd);
  s.eofft = (int *)(base + L.o_eofft);
  s.stepd = (double *)(base + L.o_stepd);
  s.stept = (double *)(base + L.o_stept);
  s.stepq = (uint64_t *)(base + L.o_stepq);
  s.thq = (uint64_t *)(base + L.o_thq);
  s.esd = (int *)(base + L.o_esd);
  s.ecls = (int *)(base + L.o_ecls);
  s.fx = (int64_t *)(base + L.o_fx);
  s.redh = (int *)(base + L.o_redh);
  s.rfm = (int *)(base + L.o_rfm);
  s.etab = etab;
  return s;
}

__device__ __forceinline__ int bit_of(const uint32_t *T, int n, int row, int col) {
  return (T[(col >> 5) * n + row] >> (col & 31)) & 1;
}

// ---------------------------------------------------------------- reductions
// Sum of V doubles over the 32 lanes of a warp by recursive halving: stage s
// exchanges half of the remaining values with the lane 16>>s away, so a lane
// does V-1 + (5 - log2 V) additions instead of 5V. Afterwards the lane holds the
// warp total of quantity q(lane) in v[0]; lanes with bit 0 clear report it.
template <int V>
__device__ __forceinline__ int warp_multi_sum(double (&v)[V], int lane) {
  int q = 0;
  int cnt = V;
#pragma unroll
  for (int s = 0; (1 << s) < V; ++s) {
    const int o = 16 >> s;
    const int half = V >> (s + 1);
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int x = 0; x < half; ++x) {
      const double send = up ? v[x] : v[x + half];
      const double keep = up ? v[x + half] : v[x];
      const double got = __shfl_xor_sync(kFull, send, o);
      v[x] = __dadd_rn(keep, got);
    }
    if (up) q += half;
    cnt = half;
  }
  (void)cnt;
  // remaining butterfly stages (lanes sharing a quantity)
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int o = 16 >> s;
    if ((1 << s) >= V) v[0] = __dadd_rn(v[0], __shfl_xor_sync(kFull, v[0], o));
  }
  return q;
}

__device__ __forceinline__ long long warp_max_ll(long long x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    long long y = __shfl_xor_sync(kFull, x, o);
    x = y > x ? y : x;
  }
  return x;
}

__device__ __forceinline__ long long warp_sum_ll(long long x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
  return x;
}

// Team-wide helpers. `red` is the team's scratch (>= 32*G doubles).
__device__ __forceinline__ long long team_max_ll(const Team &T, long long x, double *red) {
  x = warp_max_ll(x);
  if (T.G == 1) return x;
  long long *r = (long long *)red;
  T.sync();
  if (T.lane == 0) r[T.warp] = x;
  T.sync();
  long long m = r[0];
  for (int w = 1; w < T.G; ++w) m = r[w] > m ? r[w] : m;
  return m;
}

__device__ __forceinline__ long long team_sum_ll(const Team &T, long long x, double *red) {
  x = warp_sum_ll(x);
  if (T.G == 1) return x;
  long long *r = (long long *)red;
  T.sync();
  if (T.lane == 0) r[T.warp] = x;
  T.sync();
  long long m = 0;
  for (int w = 0; w < T.G; ++w) m += r[w];
  return m;
}

// Argmax of (key, -j) over the team: larger key wins, ties to the smaller j.
__device__ __forceinline__ int team_argmax(const Team &T, long long key, int j, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    long long k2 = __shfl_xor_sync(kFull, key, o);
    int j2 = __shfl_xor_sync(kFull, j, o);
    if (k2 > key || (k2 == key && j2 < j)) { key = k2; j = j2; }
  }
  if (T.G == 1) return j;
  long long *rk = (long long *)red;
  int *rj = (int *)(red + T.G);
  T.sync();
  if (T.lane == 0) { rk[T.warp] = key; rj[T.warp] = j; }
  T.sync();
  long long bk = rk[0];
  int bj = rj[0];
  for (int w = 1; w < T.G; ++w)
    if (rk[w] > bk || (rk[w] == bk && rj[w] < bj)) { bk = rk[w]; bj = rj[w]; }
  return bj;
}

// ------------------------------------------------------- change statistics
// Multi-network teams: network w's rows are rows + w*row_stride words, its
// in-rows cols + w*col_stride words, its count matrices cm + w*cm_stride.
struct NetBase {
  const uint32_t *rows, *cols;
  uint16_t *cm;
  size_t row_stride, col_stride, cm_stride;
  // the networks' slices' misc words (largest degrees), misc_stride apart
  const int *misc;
  size_t misc_stride;
  int D;
};

// Per-ministep context shared by all alters (uniform over the team).
struct StepCtx {
  int i, od_i, id_i, rdeg_i;
  double zvi;
  int64_t f0;   // part of the fixed-point predictor that no alter changes
  const uint64_t *tabq;
  NetBase net;
};

// Popcount of (A_word(a) & B_word(b)) summed over the W words.
__device__ __forceinline__ int pc2(const uint32_t *A, int a, const uint32_t *B, int b, int n, int W) {
  int c = 0;
  for (int w = 0; w < W; ++w) c += __popc(A[w * n + a] & B[w * n + b]);
  return c;
}

// ------------------------------------------------------- two-path counters
// Position of counter c among the counters held as matrices.
__device__ __forceinline__ int cm_rank(unsigned mask, int c) {
  return __popc(mask & ((1u << c) - 1u));
}

// Row words of a relation's transpose (for alter j, the h with the relation).
__device__ __forceinline__ const uint32_t *rel_rows(const Slice &S, const NetBase &N, int m) {
  return m == CM_ROWS ? S.cols
                      : (m == CM_COLS ? S.rows : N.rows + (size_t)(m - CM_NCOLS) * N.row_stride);
}

// Where focal actor i's counts of one counter come from: row i of its matrix (cm),
// or popcounts of the set A (and B, bs words apart) with the alters' rows in M1
// (and M2). Resolved once for a loop over the alters.
struct CountRow {
  const uint16_t *cm;
  const uint32_t *A, *B, *M1, *M2;
  int bs;
};
__device__ __forceinline__ CountRow count_row(const DevProblem &P, const Slice &S,
                                              const StepCtx &X, int n, int W, int c) {
  CountRow R{nullptr, S.rows + X.i, nullptr, nullptr, nullptr, n};
  const unsigned mask = P.cnt.mask;
  if ((mask >> c) & 1u) {
    R.cm = S.cm + cm_rank(mask, c) * cm_size(n) + (size_t)X.i * n;
    return R;
  }
  const int list = P.cnt.list[c], m1 = P.cnt.m1[c], m2 = P.cnt.m2[c];
  if (list == CL_IN) R.A = S.cols + X.i;
  else if (list == CL_MUTUAL) R.B = S.cols + X.i;
  else if (list == CL_TP0 || list == CL_TP1) {   // the transTies masks are W words
    R.B = S.tpeq + (list == CL_TP1 ? W : 0);
    R.bs = 1;
  } else if (list >= CL_NET) R.A = X.net.rows + (size_t)(list - CL_NET) * X.net.row_stride + X.i;
  R.M1 = rel_rows(S, X.net, m1);
  if (m2 != CM_NONE) R.M2 = rel_rows(S, X.net, m2);
  return R;
}
// Alter j's count.
__device__ __forceinline__ int count_of(const CountRow &R, int n, int W, int j) {
  if (R.cm) return R.cm[j];
  int c = 0;
  if (!R.B && !R.M2) {
#pragma unroll 4
    for (int w = 0; w < W; ++w) c += __popc(R.A[w * n] & R.M1[w * n + j]);
    return c;
  }
  for (int w = 0; w < W; ++w) {
    uint32_t a = R.A[w * n];
    if (R.B) a &= R.B[w * R.bs];
    c += __popc(a & R.M1[w * n + j]);
    if (R.M2) c += __popc(a & R.M2[w * n + j]);
  }
  return c;
}
__device__ __forceinline__ int count_at(const DevProblem &P, const Slice &S, const StepCtx &X,
                                        int c, int j) {
  return count_of(count_row(P, S, X, P.n, P.W, c), P.n, P.W, j);
}

// transTies: masks {h : tp_h == 0} and {h : tp_h == 1} of the two-path counts
// tp_h = |out_i & in_h| (counter c), word-parallel via ballots.
__device__ __forceinline__ void tp_masks(const Team &T, const DevProblem &P, const Slice &S,
                                         const StepCtx &X, int n, int W, int c) {
  const CountRow R = count_row(P, S, X, n, W, c);
  for (int hb = 32 * T.warp; hb < W * 32; hb += T.L) {
    const int h = hb + T.lane;
    // (a matrix's diagonal is not kept up; the actor itself counts where it has a self-tie)
    const int v = h >= n ? -1 : (R.cm && h == X.i ? pc2(S.rows, h, S.cols, h, n, W) : count_of(R, n, W, h));
    const uint32_t z0 = __ballot_sync(kFull, v == 0), z1 = __ballot_sync(kFull, v == 1);
    if (T.lane == 0) { S.tpeq[hb >> 5] = z0; S.tpeq[W + (hb >> 5)] = z1; }
  }
}

// Updates the team's count matrices for the toggle u -> v (dl = +-1) in network
// net of problem P, and for v -> u in a symmetric one: the tasks of P.cnt
// (saom_launch.h, counter_tasks), each one word of its set per lane, as many
// tasks at once as the lanes hold. The sets are read while the tie toggles: they
// hold it at most at the diagonal cell, which is left out (and never read), so
// this needs no order with the toggle. Two 16-bit counts share a word; the
// reductions need no answer, so the warp does not wait for memory, and no count
// leaves 0..2n, so no half borrows from or carries into the other.
static __device__ __noinline__ void counts_toggle(const Team &T, const DevProblem &P,
                                                  const NetBase &N, int u, int v, int dl) {
  const int n = P.n, W = P.W;
  const int lg = W > 16 ? 5 : 32 - __clz(W - 1);   // lanes per task: 2^lg
  const int per = 32 >> lg;                        // tasks per warp at a time
  for (int s = 0; s <= (P.symflag ? 1 : 0); ++s) {
    for (int t = T.warp * per + (T.lane >> lg); t < P.cnt.ntask; t += T.G * per) {
      const unsigned k = P.cnt.task[t];
      const int a = (k & 2) ? v : u, fix = (k & 4) ? v : u;
      const size_t sn = (k >> 8) & 15;
      const uint32_t *set = ((k & 1) ? N.cols + sn * N.col_stride : N.rows + sn * N.row_stride) +
                            a;
      uint16_t *M = N.cm + (size_t)(k >> 12) * N.cm_stride + ((k >> 4) & 15) * cm_size(n);
      const size_t base = (k & 8) ? fix : (size_t)fix * n, stride = (k & 8) ? n : 1;
      for (int w = T.lane & ((1 << lg) - 1); w < W; w += 32) {
        uint32_t m = set[w * n];
        if (w == (fix >> 5)) m &= ~(1u << (fix & 31));
        while (m) {
          const size_t cell = base + stride * ((w << 5) + __ffs(m) - 1);
          m &= m - 1;
          atomicAdd(reinterpret_cast<unsigned *>(M) + (cell >> 1), (unsigned)dl << (16 * (cell & 1)));
        }
      }
    }
    const int x = u;
    u = v;
    v = x;
  }
}

// Exact (double)c for 0 <= c < 2^31 built on the integer pipes.
__device__ __forceinline__ double i2d(int c) {
  if (c == 0) return 0.0;
  const int e = 31 - __clz(c);
  const unsigned long long m = ((unsigned long long)(unsigned)c << (52 - e)) & 0xFFFFFFFFFFFFFull;
  return __longlong_as_double((long long)((((unsigned long long)(1023 + e)) << 52) | m));
}
// x * delta for delta = +-1 is exact, so it is a sign flip (sgn = 0 or 1<<63).
__device__ __forceinline__ double flip(double x, unsigned long long sgn) {
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)sgn);
}

// 2^e as a double, -1022 <= e <= 1023.
__device__ __forceinline__ double pow2(int e) {
  return __longlong_as_double((long long)(1023 + e) << 52);
}
// A real magnitude in fixed point: d 2^sd + 2^62.
__device__ __forceinline__ uint64_t real_fx(double d, int sd) {
  return (uint64_t)(__double2ll_rn(__dmul_rn(d, pow2(sd))) + (1LL << 62));
}

// Generic change statistic of one effect (src/libcusna_saom_cpu.cpp:49-101 and
// :246-251): the reference formula evaluated per alter. Used for the kinds no
// table covers (gwdsp, interactions, dyadic covariates of very large n); cnt is
// the effect's two-path count of j (types 24, 26-28).
static __device__ __noinline__ double gen_stat(const DevProblem &P, const Slice &S, const StepCtx &X,
                                        int e, int j, int aij, int aji, int cnt,
                                        const double *d) {
  const int n = P.n, W = P.W, i = X.i, t = S.tid[e];
  const unsigned long long sg = aij ? 0x8000000000000000ull : 0ull;
  const double dl = aij ? -1.0 : 1.0;
  if (t == 32) {
    const int c2 = S.i2[e];
    double v = c2 < 0 ? dl : 1.0;
    v = __dmul_rn(v, __dmul_rn(d[S.i0[e]], d[S.i1[e]]));
    if (c2 >= 0) v = __dmul_rn(v, d[c2]);
    return v;
  }
  double vi = 0.0, vj = 0.0;
  if ((t >= 10 && t <= 13) || t == 20 || t == 21 || t == 25 || t == 31) {
    const bool dy = S.dyn[e] != 0;
    vi = dy ? X.zvi : P.vmat[(size_t)e * n + i];
    vj = dy ? __dsub_rn((double)S.z[j], P.zbar) : P.vmat[(size_t)e * n + j];
  }
  switch (t) {
    case 7: return flip(sqrt(i2d(S.indeg[j] + 1 - aij)), sg);
    case 9: return flip(sqrt(i2d(S.outdeg[j])), sg);
    case 24: case 26: case 27: case 28: return flip(P.wtab[(size_t)e * (n + 1) + cnt], sg);
    case 11: return flip(vj, sg);
    case 12: return flip(__dsub_rn(__dsub_rn(1.0, __dmul_rn(fabs(__dsub_rn(vi, vj)), S.p1[e])), S.p2[e]), sg);
    case 13: return flip(fabs(__dsub_rn(vi, vj)) < 1e-9 ? 1.0 : 0.0, sg);
    case 20:
      if (vi > __dadd_rn(vj, 1e-9)) return dl;
      if (fabs(__dsub_rn(vi, vj)) <= 1e-9) return flip(0.5, sg);
      return 0.0;
    case 21: return __dmul_rn(flip(vi, sg), vj);
    case 25: return flip(__dadd_rn(vi, vj), sg);
    case 31: return flip(vj >= __dsub_rn(S.p1[e], 1e-12) ? 1.0 : 0.0, sg);
    case 29: case 30: {
      // over h in out_j (29) or in_j (30), h != i, ascending h as the reference
      // adds: the gw weight difference at p_h = |out_i & in_h| (29) or
      // |out_i & out_h| (30), both precomputed for this ministep
      const double *wr = P.wtab + (size_t)e * (n + 1);
      const uint32_t *B = (t == 29) ? S.rows : S.cols;
      const int *pc = (t == 29) ? S.tp : S.tq;
      double acc = 0.0;
      for (int w = 0; w < W; ++w) {
        uint32_t m = B[w * n + j];
        if ((i >> 5) == w) m &= ~(1u << (i & 31));
        while (m) {
          const int h = (w << 5) + __ffs(m) - 1;
          m &= m - 1;
          const int p = pc[h];
          acc = __dadd_rn(acc, aij ? __dsub_rn(wr[p], wr[p - 1]) : __dsub_rn(wr[p + 1], wr[p]));
        }
      }
      return flip(acc, sg);
    }
    default: return 0.0;
  }
}

// gwdsp's magnitude at 2^sd + 2^62 (type 29, or 30) from the fixed-point weight
// differences w[p + 1] - w[p]: whole-number sums over the set bits of alter j's
// row. Float64 differences put two dependent FP64 additions on each set bit.
__device__ __forceinline__ uint64_t gw_fixed(const Slice &S, const StepCtx &X, int n, int W, int e,
                                             int t, int j, int aij) {
  const uint64_t *dq = X.tabq + S.eoffd[e] - aij;   // a tie's alter is in every p_h
  const uint32_t *B = (t == 29 ? S.rows : S.cols) + j;
  const int *pc = t == 29 ? S.tp : S.tq;
  uint64_t acc = 1ull << 62;
  for (int w = 0; w < W; ++w) {
    uint32_t m = B[w * n];
    if ((X.i >> 5) == w) m &= ~(1u << (X.i & 31));
    while (m) {
      const int h = (w << 5) + __ffs(m) - 1;
      m &= m - 1;
      acc += dq[pc[h]];
    }
  }
  return acc;
}

// Per-ministep magnitudes of the K_STEP effects (types 10, 14-19): for each
// (a_ij, a_ji) the reference's d and theta * d, into stepd/stept[e*4 + q],
// q = 2*a_ij + a_ji, and the magnitude in fixed point. Lanes take (e, q) pairs.
__device__ __forceinline__ void step_values(const Team &T, const DevProblem &P, const Slice &S,
                                            const StepCtx &X) {
  for (int x = T.tl; x < 4 * P.k; x += T.L) {
    const int e = x >> 2, q = x & 3;
    if (S.ekind[e] != K_STEP) continue;
    const int aij = q >> 1, aji = q & 1;
    const unsigned long long sg = aij ? 0x8000000000000000ull : 0ull;
    const double dl = aij ? -1.0 : 1.0;
    double v;
    switch (S.tid[e]) {
      case 10: v = flip(S.dyn[e] ? X.zvi : P.vmat[(size_t)e * P.n + X.i], sg); break;
      case 14: v = flip(i2d(X.id_i), sg); break;
      case 15: v = flip(sqrt(i2d(X.id_i)), sg); break;
      case 16: v = flip(__dadd_rn(__dmul_rn(2.0, i2d(X.od_i)), dl), sg); break;
      case 17: {
        const double d0 = i2d(X.od_i), d1 = __dadd_rn(d0, dl);
        v = __dsub_rn(__dmul_rn(d1, sqrt(d1)), __dmul_rn(d0, sqrt(d0)));
        break;
      }
      case 18: {
        const double d0 = i2d(X.od_i);
        v = __dsub_rn(fmin(__dadd_rn(d0, dl), S.p1[e]), fmin(d0, S.p1[e]));
        break;
      }
      case 19:
        v = flip(__dadd_rn(i2d(X.rdeg_i), __dmul_rn((double)aji, __dadd_rn(i2d(X.od_i), dl))), sg);
        break;
      default: v = 0.0; break;
    }
    S.stepd[x] = v;
    S.stept[x] = __dmul_rn(S.th[e], v);
    S.stepq[x] = real_fx(flip(v, sg), S.esd[e]);
  }
}

// Change statistics of toggling i -> j for all k effects into d[0..k-1]
// (src/libcusna_saom_cpu.cpp:49-101 per effect type, :243-261 for the loop with
// interactions and creation/endowment zeroing), and with TERMS the linear
// predictor f = sum_e theta_e d_e in the reference's e-order. The two-path
// counters replace the reference's O(n) dense loops; they count the same sets:
//   |out_i & in_j| = #{h: a_ih a_hj}: set out_i, ties h -> j
//   |out_i & out_j| = #{h: a_ih a_jh}: set out_i, ties j -> h
//   |out_j & in_i| = #{h: a_jh a_hi}: set in_i, ties j -> h
//   |in_i & in_j| = #{h: a_hi a_hj}: set in_i, ties h -> j
// Every d and every term equals the reference's float64 value: delta * x is a
// sign flip, table entries are the reference's expressions evaluated once, and
// f adds the terms in e-order (terms of zeroed effects are +-0 and change
// nothing, so they are skipped).
// Cross-network change statistic magnitude (before the sign of the toggle) of
// toggling i -> j in the own network for cross effect type t, reading network
// w's current rows (src/libcusna_saom_cpu.cpp:431-444): 33 a_w[i][j], 34
// a_w[j][i], 35 both, 36 |out_w(i) & out_w(j)| and 37 |out_w(i) & in_own(j)|
// (counter c).
__device__ __forceinline__ int cross_count(const DevProblem &P, const Slice &S, const StepCtx &X,
                                           int n, int t, int w, int c, int i, int j) {
  if (t >= 36) return count_at(P, S, X, c, j);
  int v = 1;
  if (t != 34) v = bit_of(X.net.rows + (size_t)w * X.net.row_stride, n, i, j);
  if (t != 33) v &= bit_of(X.net.cols + (size_t)w * X.net.col_stride, n, i, j);
  return v;
}

// MULTI: the kernel serves multi-network problems (cross effects K_CROSS);
// the single-network kernel compiles without that branch.
template <bool TERMS, bool MULTI>
__device__ __forceinline__ double change_stats(const DevProblem &P, const Slice &S,
                                               const StepCtx &X, int j, int aij, int aji,
                                               double *d) {
  const int n = P.n, k = P.k, i = X.i;
  const unsigned long long sg = aij ? 0x8000000000000000ull : 0ull;
  const bool ttab = (P.flags & F_THETA_TAB) != 0;
  double f = 0.0;
#pragma unroll 1
  for (int e = 0; e < k; ++e) {
    const int kind = S.ekind[e], pk = S.ecfn[e], cfn = pk & 0xFF;
    const int ca = (pk >> 8) & 0xFF, cb = (pk >> 16) & 0xFF, cc = (pk >> 24) & 0xFF;
    auto cnt = [&](int c) { return count_at(P, S, X, c, j); };
    (void)cb; (void)cc;
    double v, term = 0.0;
    bool has_term = TERMS;
    if (kind == K_CNT) {
      int c;
      switch (cfn) {
        case 0: c = 1; break;
        case 1: c = aji; break;
        case 2: case 3: c = cnt(ca); break;
        case 4: c = S.indeg[j] + 1 - aij; break;
        case 5: c = cnt(aij ? cb : ca) + (cnt(cc) > 0 ? 1 : 0); break;
        case 6: c = (aji ? cnt(ca) : 0) + cnt(cb); break;
        default: c = S.outdeg[j]; break;  // 7
      }
      v = flip(i2d(c), sg);
      if (TERMS) term = ttab ? flip(P.tab[S.eofft[e] + c], sg) : __dmul_rn(S.th[e], v);
    } else if (kind == K_LOOK) {
      int idx;
      switch (cfn) {
        case 4: idx = S.indeg[j] + 1 - aij; break;
        case 7: idx = S.outdeg[j]; break;
        case 8: idx = cnt(ca); break;
        case 12: idx = j; break;
        case 13: idx = S.z[j] - P.zlo; break;
        case 14: idx = i * n + j; break;
        default: idx = (S.z[i] - P.zlo) * P.zR + (S.z[j] - P.zlo); break;  // 15
      }
      v = flip(P.tab[S.eoffd[e] + idx], sg);
      if (TERMS) term = ttab ? flip(P.tab[S.eofft[e] + idx], sg) : __dmul_rn(S.th[e], v);
    } else if (kind == K_STEP) {
      const int q = 2 * aij + aji;
      v = S.stepd[4 * e + q];
      term = S.stept[4 * e + q];
    } else if (kind == K_ZERO) {
      v = 0.0;
      has_term = false;
    } else if (MULTI && kind == K_CROSS) {
      v = flip(i2d(cross_count(P, S, X, n, cfn, S.eoffd[e], ca, i, j)), sg);
      if (TERMS) term = __dmul_rn(S.th[e], v);
    } else {
      v = gen_stat(P, S, X, e, j, aij, aji, ca != 0xFF ? cnt(ca) : 0, d);
      if (TERMS) term = __dmul_rn(S.th[e], v);
    }
    if ((S.ety[e] == 1 && aij) || (S.ety[e] == 2 && !aij)) {
      v = 0.0;
      has_term = false;
    }
    d[e] = v;
    if (has_term) f = __dadd_rn(f, term);
  }
  return f;
}

// ---- the fixed-point pass -----------------------------------------------------
// How an effect enters the pass (Slice::ecls; bit 8: theta < 0):
enum : int {
  FX_ZERO = 0,   // d = 0
  FX_DELTA = 1,  // d = delta (density): part of f0, its score sum is that of delta w
  FX_UNI = 2,    // magnitude the same for every alter (egoX, in-degree effects): as above
  FX_CNT = 3,    // integer magnitude
  FX_REAL = 4,   // real magnitude
};
__host__ __device__ __forceinline__ int fx_class(int kind, int cfn, int tid, int ety) {
  if (kind == K_ZERO) return FX_ZERO;
  if (kind == K_CNT && cfn == 0 && ety == 0) return FX_DELTA;
  if (kind == K_STEP && (tid == 10 || tid == 14 || tid == 15) && ety == 0) return FX_UNI;
  return (kind == K_CNT || kind == K_CROSS) ? FX_CNT : FX_REAL;
}
// theta of a count at scale 2^-46 (a float32 of at least 2^-23 is exact), of a
// real statistic |theta| 2^(110 - sd), so that mulhi_fx with a magnitude at 2^sd
// has scale 2^-46.
__device__ __forceinline__ uint64_t theta_fx(double th, int cls, int sd) {
  if (cls == FX_UNI || cls == FX_REAL) return (uint64_t)__double2ull_rn(__dmul_rn(fabs(th), pow2(110 - sd)));
  return (uint64_t)__double2ll_rn(__dmul_rn(th, pow2(kFBits)));
}
// theta times the real magnitude m = |d| 2^sd + 2^62, but for the 2^62's part,
// which is -base_fx and enters the predictor's constant part where it can.
__device__ __forceinline__ int64_t term_fx(uint64_t thr, int cls, uint64_t m) {
  return signed_fx(mulhi_fx(thr, m), cls >> 8);
}
__device__ __forceinline__ int64_t base_fx(uint64_t thr, int cls) {
  return signed_fx(thr >> 2, (cls >> 8) ^ 1);
}

// The magnitude of a product from its components' a, b and (of three) c, each below
// 2^62 at its scale: ab 2^-62 has scale sa + sb - 62 and is shifted up to the
// product's own scale, which follows from the product of the bounds (fx_scale; at
// most 2 above), so that |theta| 2^(110 - sd) stays below 2^63 as for any other effect.
__device__ __forceinline__ uint64_t product_fx(int64_t a, int64_t b, int have, int want) {
  const int up = want > have ? (want - have < 63 ? want - have : 63) : 0;
  return (uint64_t)__mul64hi((int64_t)((uint64_t)a << 1), (int64_t)((uint64_t)b << 1)) << up;
}
__device__ __forceinline__ uint64_t product_fx(int64_t a, int64_t b, int64_t c, int have, int want) {
  return product_fx(__mul64hi((int64_t)((uint64_t)a << 1), (int64_t)((uint64_t)b << 1)), c, have, want);
}

// Magnitudes of toggling i -> j for the effects of classes FX_CNT (the count) and
// FX_REAL (|d| 2^sd + 2^62) into v, 0 for an effect that its creation or
// endowment type rules out, and the predictor without its sign (f_j = delta
// times it) at scale 2^-46. The terms' errors are at most 3 2^-46 each (mulhi_fx
// and the rounding of theta and d), 0 for counts.
template <bool MULTI>
__device__ __forceinline__ int64_t change_fixed(const DevProblem &P, const Slice &S,
                                                const StepCtx &X, int j, int aij, int aji,
                                                uint64_t *v) {
  const int n = P.n, k = P.k, i = X.i;
  uint64_t f = (uint64_t)X.f0;   // partial sums may wrap
#pragma unroll 1
  for (int e = 0; e < k; ++e) {
    const int cls = S.ecls[e] & 0xFF;
    if (cls < FX_CNT) continue;
    const int kind = S.ekind[e], pk = S.ecfn[e], cfn = pk & 0xFF;
    const int ca = (pk >> 8) & 0xFF, cb = (pk >> 16) & 0xFF, cc = (pk >> 24) & 0xFF;
    auto cnt = [&](int c) { return count_at(P, S, X, c, j); };
    const int ety = S.ety[e];
    if ((ety == 1 && aij) || (ety == 2 && !aij)) {
      v[e] = 0;
      continue;
    }
    if (cls == FX_CNT) {
      int c;
      if (MULTI && kind == K_CROSS) {
        c = cross_count(P, S, X, n, cfn, S.eoffd[e], ca, i, j);
      } else {
        switch (cfn) {
          case 0: c = 1; break;
          case 1: c = aji; break;
          case 2: case 3: c = cnt(ca); break;
          case 4: c = S.indeg[j] + 1 - aij; break;
          case 5: c = cnt(aij ? cb : ca) + (cnt(cc) > 0 ? 1 : 0); break;
          case 6: c = (aji ? cnt(ca) : 0) + cnt(cb); break;
          default: c = S.outdeg[j]; break;  // 7
        }
      }
      v[e] = (uint64_t)c;
      f += S.thq[e] * (uint32_t)c;
      continue;
    }
    uint64_t m;
    if (kind == K_LOOK) {
      int idx;
      switch (cfn) {
        case 4: idx = S.indeg[j] + 1 - aij; break;
        case 7: idx = S.outdeg[j]; break;
        case 8: idx = cnt(ca); break;
        case 12: idx = j; break;
        case 13: idx = S.z[j] - P.zlo; break;
        case 14: idx = i * n + j; break;
        default: idx = (S.z[i] - P.zlo) * P.zR + (S.z[j] - P.zlo); break;  // 15
      }
      m = X.tabq[S.eoffd[e] + idx];
    } else if (kind == K_STEP) {
      m = S.stepq[4 * e + 2 * aij + aji];
    } else if (S.tid[e] == 32) {
      // product of the components' magnitudes (each at its scale)
      auto mag = [&](int q) -> int64_t {
        const int cl = S.ecls[q] & 0xFF;
        if (cl == FX_DELTA) return (int64_t)1 << S.esd[q];
        if (cl == FX_CNT) return (int64_t)(v[q] << S.esd[q]);
        if (cl == FX_UNI) return (int64_t)(S.stepq[4 * q] + kMinus62);
        return cl == FX_REAL && v[q] ? (int64_t)(v[q] + kMinus62) : 0;
      };
      const int a = S.i0[e], b = S.i1[e], c = S.i2[e], have = S.esd[a] + S.esd[b] - 62;
      m = (c < 0 ? product_fx(mag(a), mag(b), have, S.esd[e])
                 : product_fx(mag(a), mag(b), mag(c), have + S.esd[c] - 62, S.esd[e])) +
          (1ull << 62);
    } else if (cfn == 16) {
      m = gw_fixed(S, X, n, P.W, e, S.tid[e], j, aij);
    } else {
      const double g = gen_stat(P, S, X, e, j, aij, aji, ca != 0xFF ? cnt(ca) : 0, nullptr);
      m = real_fx(aij ? -g : g, S.esd[e]);
    }
    v[e] = m;
    f += (uint64_t)term_fx(S.thq[e], S.ecls[e], m);
    if (ety) f += (uint64_t)base_fx(S.thq[e], S.ecls[e]);
  }
  return (int64_t)f;
}

// Behaviour change statistic, src/libcusna_saom_cpu.cpp:103-113.
__device__ __forceinline__ double beh_stat(int t, double dl, double zc, long long nb, double zs,
                                           long long nh, long long ne, long long nl, double br,
                                           double bs) {
  double tc;
  switch (t) {
    case 0: return dl;
    case 1: return __dmul_rn(__dadd_rn(__dmul_rn(2.0, zc), dl), dl);
    case 2: return nb > 0 ? __ddiv_rn(__dmul_rn(dl, zs), (double)nb) : 0.0;
    case 3:
      if (nb == 0) return 0.0;
      tc = dl > 0 ? (double)(nh - ne - nl) : (double)(nl - ne - nh);
      return __ddiv_rn(tc, __dmul_rn(br, (double)nb));
    case 4:
      if (nb == 0) return 0.0;
      tc = dl > 0 ? (double)(nh - ne - nl) : (double)(nl - ne - nh);
      return __dsub_rn(__ddiv_rn(tc, br), __dmul_rn((double)nb, bs));
  }
  return 0.0;
}

}  // namespace cusna
