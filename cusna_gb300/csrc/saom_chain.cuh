// saom_chain.cuh -- one chain of one period, run by a team of G warps.
// Restates src/libcusna_saom_cpu.cpp:142-303 (simulate_one) and :394-422 (the
// per-chain outputs) over bitsets.
#pragma once
#include "saom_kernel.cuh"
#include "saom_stats.cuh"

namespace cusna {

// The actor and word counts: constants where a specialised build fixes them.
__device__ __forceinline__ int prob_n(const DevProblem &P) {
#ifdef CUSNA_JIT_N
  return CUSNA_JIT_N;
#else
  return P.n;
#endif
}
__device__ __forceinline__ int prob_w(const DevProblem &P) {
#ifdef CUSNA_JIT_N
  return (CUSNA_JIT_N + 31) / 32;
#else
  return P.W;
#endif
}
__device__ __forceinline__ int prob_k(const DevProblem &P) {
#ifdef CUSNA_JIT_K
  return CUSNA_JIT_K;
#else
  return P.k;
#endif
}

// exp_fx's table into the CTA's shared memory (every thread of the CTA calls).
__device__ __forceinline__ void load_exp_table(int2 *etab, const DevProblem *probs) {
  const int2 *src = reinterpret_cast<const int2 *>(probs[0].tabq);
  for (int x = threadIdx.x; x < 256; x += blockDim.x) etab[x] = src[x];
  __syncthreads();
}

// Fixed-point scales, classes and parameters (one lane). The pass over the alters
// needs every |f_j| < 2^14, by bounds on the statistics: of the own network's counts
// and degrees a cap, S.fx[2], which starts as what n allows and is halved until the
// parameters fit, while it is above the counts that the chain starts with (mb). A
// chain that nears its cap (cap_check), or that none fits, runs in float64
// (S.fx[1] = 0). With the bounds of n alone, chains of large sparse networks did from
// the start: transTrip's at n = 8192 alone allowed |theta| < 1.
__device__ __forceinline__ void chain_scales(const DevProblem &P, const Slice &S, int mb) {
  const int k = prob_k(P);
  double range = 0.0;
  int cap = max(16, 2 * P.n + 2);
  for (;; cap /= 2) {
    range = 0.0;
    for (int e = 0; e < k; ++e) {
      const int kind = S.ekind[e], t = S.tid[e];
      const int cls = fx_class(kind, S.ecfn[e] & 0xFF, t, S.ety[e]);
      double bound = P.ebound[e];
      if (kind == K_CNT || (kind == K_STEP && t >= 14 && t <= 19 && t != 18))
        bound = bound > (double)cap ? (double)cap : bound;
      if (t == 32 && kind != K_ZERO) {   // products: the components' bounds
        bound = __dmul_rn(S.dstar[S.i0[e]], S.dstar[S.i1[e]]);
        if (S.i2[e] >= 0) bound = __dmul_rn(bound, S.dstar[S.i2[e]]);
      }
      S.dstar[e] = bound;
      S.esd[e] = fx_scale(bound);
      S.ecls[e] = cls | (S.th[e] < 0.0 ? 256 : 0);
      // (scales of bounds beyond these powers of ten would leave pow2's range)
      const bool scaled = bound == 0.0 || (bound >= 1e-250 && bound <= 1e250);
      if (cls != FX_ZERO)
        range = __dadd_rn(range, scaled ? __dmul_rn(fabs(S.th[e]), bound) : (double)INFINITY);
    }
    if (range < 16384.0 || !(cap / 2 >= mb)) break;
  }
  uint64_t f0 = 0;
  const bool in_range = range < 16384.0;      // false for a NaN
  if (in_range)
    for (int e = 0; e < k; ++e) {
      S.thq[e] = theta_fx(S.th[e], S.ecls[e] & 0xFF, S.esd[e]);
      if ((S.ecls[e] & 0xFF) == FX_DELTA) f0 += S.thq[e];
      // the part of a real magnitude's 2^62, for every alter alike
      if ((S.ecls[e] & 0xFF) == FX_UNI || ((S.ecls[e] & 0xFF) == FX_REAL && S.ety[e] == 0))
        f0 += (uint64_t)base_fx(S.thq[e], S.ecls[e]);
    }
  S.fx[0] = (int64_t)f0;
  S.fx[1] = in_range;
  S.fx[2] = cap >= 2 * P.n + 2 ? 0x7FFFFFFF : cap;
  S.misc[15] = in_range;
}

// Before every 32nd ministep (one lane): whether the next 32 toggles keep the counts
// and degrees below the cap.
constexpr int kCapEvery = 32;
__device__ __forceinline__ int capped_counts(int max_out, int max_in) {
  return max(16, max(2 * (max_out + kCapEvery) + 2, max_in + kCapEvery + 1));
}
__device__ __forceinline__ void cap_check(const Slice &S) {
  if (capped_counts(S.misc[11], S.misc[10]) > (int)S.fx[2]) S.fx[1] = 0;
}

// Load the chain's start state and parameters into the team slice.
__device__ __forceinline__ void chain_init(const Team &T, const DevProblem &P, const Slice &S,
                                           int c) {
  const int n = P.n, W = P.W, k = P.k, L = T.L;
  for (int x = T.tl; x < W * n; x += L) {
    S.rows[x] = P.simr[x];
    S.cols[x] = P.simc[x];
  }
  for (int e = T.tl; e < k; e += L) {
    S.th[e] = (double)P.theta[(size_t)c * P.prow * k + e];
    S.sc[e] = 0.0;
    S.tid[e] = P.type_ids[e];
    S.ety[e] = P.etypes[e];
    S.dyn[e] = P.dyn[e];
    S.i0[e] = P.int0[e];
    S.i1[e] = P.int1[e];
    S.i2[e] = P.int2[e];
    S.p1[e] = P.p1[e];
    S.p2[e] = P.p2[e];
    S.ekind[e] = P.ekind[e];
    S.ecfn[e] = P.ecfn[e];
    S.eoffd[e] = P.eoffd[e];
    S.eofft[e] = P.eofft[e];
  }
  for (int e = T.tl; e < P.kb; e += L) {
    S.thb[e] = P.thetab ? (double)P.thetab[(size_t)c * P.prow * P.kb + e] : 0.0;
    S.bsc[e] = 0.0;
    S.bty[e] = P.bty[e];
  }
  for (int q = T.tl; q < P.nrate; q += L) {
    S.rsc[q] = 0.0;
    S.rkind[q] = P.rkind[q];
  }
  if (P.cnt.mask) {
    // the count matrices' start values, 16 bytes per access
    const size_t words = __popc(P.cnt.mask) * cm_size(n) / 8;
    const uint4 *src = reinterpret_cast<const uint4 *>(P.c0);
    uint4 *dst = reinterpret_cast<uint4 *>(S.cm);
    size_t x = T.tl;
    for (; x + 3 * (size_t)L < words; x += 4 * (size_t)L) {
      const uint4 a = src[x], b = src[x + L], c4 = src[x + 2 * L], e4 = src[x + 3 * L];
      dst[x] = a;
      dst[x + L] = b;
      dst[x + 2 * L] = c4;
      dst[x + 3 * L] = e4;
    }
    for (; x < words; x += L) dst[x] = src[x];
  }
  if (P.flags & F_HAS_Z)
    for (int x = T.tl; x < n; x += L) S.z[x] = P.z0[x];
  if (P.nrate > 0)
    for (int x = T.tl; x < n; x += L) S.crate[x] = 1.0;
  if (T.tl == 0) S.misc[13] = c;   // the chain's index within its problem (validation words)
  T.sync();
  for (int x = T.tl; x < n; x += L) {
    int od = 0, id = 0;
    for (int w = 0; w < W; ++w) {
      od += __popc(S.rows[w * n + x]);
      id += __popc(S.cols[w * n + x]);
    }
    S.outdeg[x] = od;
    S.indeg[x] = id;
  }
  T.sync();
  // largest degrees, kept up (never lowered) by the toggles: the bound on a
  // count in step_guard
  int mo = 0, mi = 0;
  for (int x = T.tl; x < n; x += L) {
    mo = max(mo, (int)S.outdeg[x]);
    mi = max(mi, (int)S.indeg[x]);
  }
  mo = (int)team_max_ll(T, mo, S.red);
  mi = (int)team_max_ll(T, mi, S.red);
  if (T.tl == 0) {
    S.misc[10] = mi;
    S.misc[11] = mo;
    chain_scales(P, S, capped_counts(mo, mi));
  }
  T.sync();
}

// Per-ministep helper arrays: transTies masks, gwdsp counts as integers per
// actor. Complete for the whole team on return.
__device__ __forceinline__ void step_helpers(const Team &T, const DevProblem &P, const Slice &S,
                                             const StepCtx &X) {
  const int n = prob_n(P), W = prob_w(P), fl = P.flags;
  if (fl & F_NEED_TP) tp_masks(T, P, S, X, n, W, P.cnt.tp);
  if (fl & F_NEED_GW29) {
    const CountRow R = count_row(P, S, X, n, W, P.cnt.tp);
    for (int h = T.tl; h < n; h += T.L) S.tp[h] = count_of(R, n, W, h);
  }
  if (fl & F_NEED_GW30) {
    const CountRow R = count_row(P, S, X, n, W, P.cnt.tq);
    for (int h = T.tl; h < n; h += T.L) S.tq[h] = count_of(R, n, W, h);
  }
  if (fl & (F_NEED_TP | F_NEED_GW29 | F_NEED_GW30)) T.sync();
}

// The four Philox words of ministep ms, counter (ms, chain, 0, 0) as the
// reference draws them (src/libcusna_saom_cpu.cpp:167); in validation mode
// (VALID) the caller's words for that ministep while they last.
template <bool VALID>
__device__ __forceinline__ void step_words(const DevProblem &P, const Slice &S, long long ms,
                                           uint32_t chain, uint32_t out[4]) {
  if (VALID && P.ustream && ms < P.ustream_steps) {
    const uint32_t *u =
        P.ustream + ((size_t)S.misc[13] * P.ustream_steps + (size_t)ms) * (4 + (size_t)P.n);
    out[0] = u[0]; out[1] = u[1]; out[2] = u[2]; out[3] = u[3];
    return;
  }
  philox10((uint32_t)ms, chain, 0u, 0u, P.k0, P.k1, out);
}

// The Gumbel word of alter j in ministep ms: first output of counter
// (ms, chain, 1, j) (src/libcusna_saom_cpu.cpp:266), or the caller's word.
template <bool VALID>
__device__ __forceinline__ uint32_t alter_word(const DevProblem &P, const Slice &S, long long ms,
                                               uint32_t chain, int j, uint32_t k0, uint32_t k1) {
  if (VALID && P.ustream && ms < P.ustream_steps)
    return P.ustream[((size_t)S.misc[13] * P.ustream_steps + (size_t)ms) * (4 + (size_t)P.n) + 4 +
                     (size_t)j];
  uint32_t ph[4];
  philox10((uint32_t)ms, chain, 1u, (uint32_t)j, k0, k1, ph);
  return ph[0];
}

// Behaviour ministep (src/libcusna_saom_cpu.cpp:202-227), run by the team's first
// warp: the reference's operations and order of sums, with what does not depend on
// one another side by side (the row's words, the neighbours' values, the effects'
// statistics up and down, the exponentials, the divisions). Bound by the chain of
// dependent FP64 operations that is left (by one lane, 1024 co-evolution chains of
// 1000 actors took 194 ms instead of 156). Updates z, bsc, *bdist; returns the step
// d in {-1, 0, 1}.
static __device__ int beh_step(const Team &T, const DevProblem &P, const Slice &S, int i,
                               uint32_t r3, long long *bdist) {
  const int n = P.n, W = P.W, kb = P.kb, lane = T.lane;
  const int zi = S.z[i];
  const double zc = __dsub_rn((double)zi, P.zbar);
  // the neighbours' values in ascending order
  int *zl = reinterpret_cast<int *>(S.gbuf);
  int cnt = 0;
  for (int w0 = 0; w0 < W; w0 += 32) {
    uint32_t m = w0 + lane < W ? S.rows[(w0 + lane) * n + i] : 0u;
    int upto = __popc(m);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, upto, o);
      if (lane >= o) upto += y;
    }
    int pos = cnt + upto - __popc(m);
    while (m) {
      zl[pos++] = S.z[((w0 + lane) << 5) + __ffs(m) - 1];
      m &= m - 1;
    }
    cnt += __shfl_sync(kFull, upto, 31);
  }
  __syncwarp();
  double zs = 0.0;
  int h = 0, q = 0;
  for (int b = 0; b < cnt; b += 32) {
    const bool on = b + lane < cnt;
    const int zj = on ? zl[b + lane] : 0;
    const double v = on ? __dsub_rn((double)zj, P.zbar) : 0.0;
    h += __popc(__ballot_sync(kFull, on && zj > zi));
    q += __popc(__ballot_sync(kFull, on && zj == zi));
    for (int x = 0; x < 32 && b + x < cnt; ++x) zs = __dadd_rn(zs, __shfl_sync(kFull, v, x));
  }
  const long long nb = cnt, nh = h, ne = q, nl = cnt - h - q;
  const bool up = zi < P.zmax, dn = zi > P.zmin;
  // lane e: effect e up, lane 8 + e: down (at most 8 effects)
  const int e = lane & 7;
  const double c = e < kb ? beh_stat(S.bty[e], lane & 8 ? -1.0 : 1.0, zc, nb, zs, nh, ne, nl,
                                     P.brange, P.bsimmean)
                          : 0.0;
  const double term = e < kb ? __dmul_rn(S.thb[e], c) : 0.0;
  double fu = 0.0, fd = 0.0;
  for (int x = 0; x < kb; ++x) {
    fu = __dadd_rn(fu, __shfl_sync(kFull, term, x));
    fd = __dadd_rn(fd, __shfl_sync(kFull, term, 8 + x));
  }
  double mx = 0.0;
  if (up && fu > mx) mx = fu;
  if (dn && fd > mx) mx = fd;
  // lane 0 down, 1 stay, 2 up
  double ex = exp(lane == 0 ? __dsub_rn(fd, mx) : (lane == 1 ? -mx : __dsub_rn(fu, mx)));
  if ((lane == 0 && !dn) || (lane == 2 && !up)) ex = 0.0;
  double pd = __shfl_sync(kFull, ex, 0), p0 = __shfl_sync(kFull, ex, 1),
         pu = __shfl_sync(kFull, ex, 2);
  const double ps = __dadd_rn(__dadd_rn(pd, p0), pu);
  ex = __ddiv_rn(ex, ps);
  pd = __shfl_sync(kFull, ex, 0);
  p0 = __shfl_sync(kFull, ex, 1);
  pu = __shfl_sync(kFull, ex, 2);
  const double uc = unif01(r3);
  const int d = uc < pd ? -1 : (uc < __dadd_rn(pd, p0) ? 0 : 1);
  const double cdn = __shfl_sync(kFull, c, 8 + e);
  if (lane < kb) {
    double s = d == 1 ? c : (d == -1 ? cdn : 0.0);
    if (up) s = __dsub_rn(s, __dmul_rn(pu, c));
    if (dn) s = __dsub_rn(s, __dmul_rn(pd, cdn));
    S.bsc[e] = __dadd_rn(S.bsc[e], s);
  }
  if (d != 0) {
    if (P.bkdist[i]) {
      const long long z0 = P.z0[i];
      long long a = (long long)(zi + d) - z0, b = (long long)zi - z0;
      *bdist += (a < 0 ? -a : a) - (b < 0 ? -b : b);
    }
    if (lane == 0) S.z[i] = zi + d;
  }
  return d;
}

// Non-basic rate draw (src/libcusna_saom_cpu.cpp:170-193). The actor rates are
// computed in parallel; lane 0 then forms S0, the rate-score sums and the focal
// actor in the reference's sequential order. Returns the focal actor, or -1
// when an unconditional period ends.
static __device__ int rate_draw(const Team &T, const DevProblem &P, const Slice &S, const uint32_t rr[4],
                         double lam, double &t, double &rho) {
  const int n = P.n, nr = P.nrate;
  for (int idx = T.tl; idx < P.nact; idx += T.L) {
    const int a2 = P.act[idx];
    double s = 0.0;
    for (int q = 0; q < nr; ++q) {
      const int rk = S.rkind[q];
      const double u = rk == 0 ? P.ru[(size_t)q * n + a2]
                               : (rk == 1 ? (double)S.outdeg[a2] : (double)S.indeg[a2]);
      s = __dadd_rn(s, __dmul_rn(P.ralpha[q], u));
    }
    if (s > 30.0) s = 30.0; else if (s < -30.0) s = -30.0;
    S.crate[a2] = exp(s);
  }
  T.sync();
  int focal = -1;
  if (T.tl == 0) {
    double S0 = 0.0, rs[4] = {0.0, 0.0, 0.0, 0.0};
    for (int idx = 0; idx < P.nact; ++idx) {
      const int a2 = P.act[idx];
      const double cc = S.crate[a2];
      S0 = __dadd_rn(S0, cc);
      for (int q = 0; q < nr; ++q) {
        const int rk = S.rkind[q];
        const double u = rk == 0 ? P.ru[(size_t)q * n + a2]
                                 : (rk == 1 ? (double)S.outdeg[a2] : (double)S.indeg[a2]);
        rs[q] = __dadd_rn(rs[q], __dmul_rn(cc, u));
      }
    }
    const double tau = __ddiv_rn(-log(unif01(rr[0])), __dmul_rn(lam, S0));
    double tau_eff = tau;
    if (!P.cond && __dadd_rn(t, tau) > 1.0) tau_eff = __dsub_rn(1.0, t);
    rho = __dadd_rn(rho, __dmul_rn(tau_eff, S0));
    for (int q = 0; q < nr; ++q)
      S.rsc[q] = __dsub_rn(S.rsc[q], __dmul_rn(__dmul_rn(tau_eff, lam), rs[q]));
    t = __dadd_rn(t, tau);
    if (!P.cond && t > 1.0) {
      focal = -1;
    } else {
      const double tgt = __dmul_rn(unif01(rr[2]), S0);
      double acc = 0.0;
      focal = P.act[P.nact - 1];
      for (int idx = 0; idx < P.nact; ++idx) {
        acc = __dadd_rn(acc, S.crate[P.act[idx]]);
        if (acc >= tgt) { focal = P.act[idx]; break; }
      }
    }
    S.misc[0] = focal;
    ((double *)(S.misc + 2))[0] = t;
    ((double *)(S.misc + 4))[0] = rho;
  }
  T.sync();
  focal = S.misc[0];
  t = ((double *)(S.misc + 2))[0];
  rho = ((double *)(S.misc + 4))[0];
  T.sync();
  return focal;
}

// Best float32 Gumbel key b1 at alter j1 with its error bound e1, and the
// largest upper bound (key + its error bound) of every other alter. The
// float32 keys certify the choice when b1 - e1 > ub2.
struct KeyTop {
  float b1, e1, ub2;
  int j1;
};
// alters reach a lane in ascending j: a key equal to the best is not better
// (its upper bound then reaches b1, which sends the choice to float64). A NaN
// key or bound (float32 overflow, or non-finite inputs) certifies nothing: it
// raises ub2 to infinity, so the exact float64 keys decide.
__device__ __forceinline__ void keytop_add(KeyTop &t, float g, float E, int j) {
  if (g > t.b1) {
    t.ub2 = fmaxf(t.ub2, __fadd_rn(t.b1, t.e1));
    t.b1 = g;
    t.e1 = E;
    t.j1 = j;
  } else {
    const float u = __fadd_rn(g, E);
    t.ub2 = (u != u) ? INFINITY : fmaxf(t.ub2, u);
  }
}
__device__ __forceinline__ void keytop_merge(KeyTop &a, const KeyTop &c) {
  if (c.b1 > a.b1 || (c.b1 == a.b1 && c.j1 < a.j1)) {
    a.ub2 = fmaxf(fmaxf(a.ub2, c.ub2), __fadd_rn(a.b1, a.e1));
    a.b1 = c.b1;
    a.e1 = c.e1;
    a.j1 = c.j1;
  } else {
    a.ub2 = fmaxf(fmaxf(a.ub2, c.ub2), __fadd_rn(c.b1, c.e1));
  }
}
// Order-preserving integer image of a float32 (no NaN), and back.
__device__ __forceinline__ int fkey(float x) {
  const int b = __float_as_int(x);
  return b ^ ((b >> 31) & 0x7FFFFFFF);
}
__device__ __forceinline__ float funkey(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7FFFFFFF)); }

// The warp's KeyTop: two integer warp maxima. Every lane other than the best
// one's contributes its own best key's upper bound; a second lane with an equal
// key then has an upper bound above it, which sends the choice to float64.
__device__ __forceinline__ KeyTop warp_keytop(const KeyTop &x, int lane) {
  const int mine = fkey(x.b1), m = __reduce_max_sync(kFull, mine);
  const int src = __ffs(__ballot_sync(kFull, mine == m)) - 1;
  const float u = lane == src ? x.ub2 : fmaxf(x.ub2, __fadd_rn(x.b1, x.e1));
  KeyTop t;
  t.ub2 = funkey(__reduce_max_sync(kFull, fkey(u)));
  t.b1 = funkey(m);
  t.e1 = __shfl_sync(kFull, x.e1, src);
  t.j1 = __shfl_sync(kFull, x.j1, src);
  return t;
}

__device__ __forceinline__ bool is_nan64(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return ((b >> 52) & 0x7FF) == 0x7FF && (b & 0xFFFFFFFFFFFFFull) != 0;
}

// The float64 predictor f_j of alter j (and its change statistics in d): the
// reference's value bit for bit (effect order, separately rounded products
// and sums).
template <bool MULTI>
__device__ __forceinline__ double f64_of(const DevProblem &P, const Slice &S, const StepCtx &X,
                                         int j, double *d, int net) {
  const int n = P.n, i = X.i;
  const int aij = bit_of(S.rows, n, i, j), aji = bit_of(S.cols, n, i, j);
  (void)net;
#if defined(CUSNA_JIT_SPEC)
  return jit_change_stats<true>(P, S, X, j, aij, aji, d);
#elif defined(CUSNA_JIT_MULTI)
  return jit_change_stats<true>(net, P, S, X, j, aij, aji, d);
#else
  return change_stats<true, MULTI>(P, S, X, j, aij, aji, d);
#endif
}

// The score sums in float64 as the reference forms them
// (src/libcusna_saom_cpu.cpp:271-274): lmax = the largest predictor of a
// permitted alter (at least the "no change" alter's 0), then sume = sum of
// exp(f_j - lmax) and wsum_e = sum of exp(f_j - lmax) d_je over permitted
// alters, every f_j and d_je the reference's float64 value. The sums run per
// 32-alter block (fixed warp reduction), every 32nd block's in order, then over
// those 32, so they do not depend on the team size; quantity 0 (the weights) and
// 1 + e land in S.red[32G + q]. Then score_e += d_{jstar,e} - wsum_e / sume. Used
// by chains whose parameters exceed the fixed-point range, by ministeps with a sum
// of few bits (sums_short), and at every ministep under F_LSE64. Called by the whole team.
template <bool MULTI, int VQ>
static __device__ __noinline__ void lse_float64(const Team T, const DevProblem &P, const Slice S,
                                                const StepCtx X, double *d, int net, int jstar) {
  constexpr int V = VQ <= 8 ? 8 : (VQ <= 16 ? 16 : 32);  // warp_multi_sum's power of two
  const int n = P.n, k = P.k, L = T.L, i = X.i;
  double *rec = reinterpret_cast<double *>(S.ring + ring_bytes(k));
  long long mk = dkey(0.0);
  for (int j = T.tl; j < n; j += L) {
    if (j == i || !((S.okbits[j >> 5] >> (j & 31)) & 1u)) continue;
    const double f = f64_of<MULTI>(P, S, X, j, d, net);
    if (!is_nan64(f)) {
      const long long kf = dkey(f);
      mk = kf > mk ? kf : mk;
    }
  }
  const double lmax = dunkey(team_max_ll(T, mk, S.red));
  for (int jb = 32 * T.warp; jb < n; jb += L) {
    const int j = jb + T.lane;
    double w = 0.0;
    bool weighted = false;
    if (j < n && ((S.okbits[j >> 5] >> (j & 31)) & 1u)) {
      if (j == i) {
        w = exp(-lmax);
      } else {
        w = exp(__dsub_rn(f64_of<MULTI>(P, S, X, j, d, net), lmax));
        weighted = true;
      }
    }
    double v[V];
    v[0] = w;
#pragma unroll
    for (int q = 1; q < V; ++q) v[q] = (weighted && q - 1 < k) ? __dmul_rn(w, d[q - 1]) : 0.0;
    const int q = warp_multi_sum<V>(v, T.lane);
    const bool writer = (V >= 32) || ((T.lane & ((32 / V) - 1)) == 0);
    if (writer && q <= k) {   // block b and b + 32 are the same warp's and lane's
      double *r = rec + ((jb >> 5) & 31) * (k + 1) + q;
      *r = jb < 1024 ? v[0] : __dadd_rn(*r, v[0]);
    }
  }
  T.sync();
  if (T.warp == 0) {
    double v[V];
#pragma unroll
    for (int q = 0; q < V; ++q)
      v[q] = q <= k && T.lane < ((n + 31) >> 5) ? __dadd_rn(0.0, rec[T.lane * (k + 1) + q]) : 0.0;
    const int q = warp_multi_sum<V>(v, T.lane);
    const bool writer = (V >= 32) || ((T.lane & ((32 / V) - 1)) == 0);
    if (writer && q <= k) S.red[32 * T.G + q] = v[0];
  }
  // the chosen alter's statistics and the score update
  if (T.tl == 0) {
    if (jstar == i)
      for (int e = 0; e < k; ++e) d[e] = 0.0;
    else
      f64_of<MULTI>(P, S, X, jstar, d, net);
    for (int e = 0; e < k; ++e) S.dstar[e] = d[e];
  }
  T.sync();
  for (int e = T.tl; e < k; e += L)
    S.sc[e] = __dadd_rn(S.sc[e], __dsub_rn(S.dstar[e], __ddiv_rn(S.red[32 * T.G + 1 + e], S.red[32 * T.G])));
}

// ---- score sums in fixed point ---------------------------------------------------
// Quantities: 0 the weights w_j (every permitted alter, "no change" included), 1
// delta_j w_j, 2 + e the weighted magnitude delta_j w_j |d_je| of an effect of
// class FX_CNT or FX_REAL. Each lane adds its alters in 64-bit integers (scale
// 2^-(44 - sh); real statistics as mulround_fx(w 2^6, m)), the warp adds its lanes'
// accumulators as three integer limbs, and the warps' sums are added as integers:
// no order matters. kFxRoom bounds a lane's sums (see step_guard).
// A specialised build fixes the number (CUSNA_FX_V) and the ones in use.
#ifndef CUSNA_FX_MASK
#define CUSNA_FX_MASK 0xFFFFFFFFu
#endif

// Adds alter j's weight W and magnitudes v to the lane's accumulators.
template <int V>
__device__ __forceinline__ void sums_add(const Slice &S, int k, uint64_t (&acc)[V], uint64_t W,
                                         int aij, const uint64_t *v) {
  const uint64_t wd = (uint64_t)signed_fx(W, aij);
  const uint64_t w6 = W << 6;
  acc[0] += W;
  acc[1] += wd;
#pragma unroll
  for (int e = 0; e < V - 2; ++e) {
    if (e >= k) continue;
    const int cls = S.ecls[e] & 0xFF;
    if (cls == FX_CNT) {
      acc[2 + e] += wd * v[e];
    } else if (cls == FX_REAL) {
      acc[2 + e] += (uint64_t)signed_fx(mulround_fx(w6, v[e]), aij);
    }
  }
}

// The warp's sums: afterwards lane q holds quantity q's total as lo + 2^48 hi.
template <int V>
__device__ __forceinline__ void sums_reduce(const uint64_t (&acc)[V], int lane, int64_t &lo, int &hi) {
  lo = 0;
  hi = 0;
#pragma unroll
  for (int q = 0; q < V; ++q) {
    if (!((CUSNA_FX_MASK >> q) & 1u)) continue;
    const uint64_t a = acc[q];
    const unsigned s0 = __reduce_add_sync(kFull, (unsigned)a & 0xFFFFFFu);
    const unsigned s1 = __reduce_add_sync(kFull, (unsigned)(a >> 24) & 0xFFFFFFu);
    const int s2 = __reduce_add_sync(kFull, (int)((int64_t)a >> 48));
    if (lane == q) {
      lo = (int64_t)s0 + ((int64_t)s1 << 24);
      hi = s2;
    }
  }
}

// The ring: ministep slot's score sums as they left the pass (quantity q as lo +
// 2^48 hi), the chosen alter's magnitudes (v of change_fixed; a FX_UNI effect's
// float64 magnitude) and meta = 4 sh + 2 a_ij + ("no change" chosen), -1 where the
// ministep's scores were formed in float64. Divisions
// and float64 arithmetic wait for scores_flush: on this chip a dependent FP64
// operation is tens of cycles and a division hundreds, 2,700 of the 8,800 cycles
// of a ministep of one warp (n = 50) when every ministep did its own; eight at
// a time, one per lane group, they cost about a tenth of that.
struct ScoreRing {
  int64_t *lo, *dst;
  int *hi, *meta;
};
__device__ __forceinline__ ScoreRing ring_of(const Slice &S, int k) {
  ScoreRing R;
  R.lo = reinterpret_cast<int64_t *>(S.ring);
  R.dst = R.lo + kRing * (k + 2);
  R.hi = reinterpret_cast<int *>(R.dst + kRing * k);
  R.meta = R.hi + kRing * (k + 2);
  return R;
}

// The "no change" alter's weight (exp_fx(0, sh)).
__device__ __forceinline__ int64_t stay_weight(int sh) {
  return sh <= kWBits ? 1LL << (kWBits - sh) : (sh == kWBits + 1 ? 1 : 0);
}
// The ring's sum at index x in float64.
__device__ __forceinline__ double count_sum(const ScoreRing &R, int x) {
  return __dadd_rn((double)R.lo[x], __dmul_rn((double)R.hi[x], 281474976710656.0));
}
// Quantity q's sum of the slot at x; of a real statistic (real) of creation or
// endowment type ty less the 2^62 of every magnitude, which added 16 w delta: over
// all alters, or over those that the creation (no tie) or endowment (tie) type
// leaves, which is half of w (1 + delta), or of w (delta - 1), without "no change"
// (stay: its weight). Taken off in integers, so that magnitudes of 0 leave 0.
__device__ __forceinline__ double sum_value(const ScoreRing &R, int x, int q, bool real, int ty,
                                            int64_t stay) {
  if (!real) return count_sum(R, x + q);
  int64_t minus8;   // a factor that the compiler does not turn into a subtraction (see signed_fx)
  asm volatile("mov.b64 %0, -8;" : "=l"(minus8));
  const int64_t cd = ty == 0 ? 2 : 1, cw = ty == 1 ? 1 : (ty == 2 ? -1 : 0),
                cs = ty == 1 ? -1 : (ty == 2 ? 1 : 0);
  int64_t lo = R.lo[x + q] + (R.lo[x + 1] * cd + R.lo[x] * cw + stay * cs) * minus8;
  const int64_t hi = R.hi[x + q] + (R.hi[x + 1] * cd + R.hi[x] * cw) * minus8 + (lo >> 48);
  lo &= (1LL << 48) - 1;
  return __dadd_rn((double)lo, __dmul_rn((double)hi, 281474976710656.0));
}

// Adds the warps' sums into the ring (one warp, lane q).
__device__ __forceinline__ void sums_combine(const Team &T, const Slice &S, const ScoreRing &R,
                                             int k, int slot) {
  const int64_t *lo = reinterpret_cast<const int64_t *>(S.red);
  int64_t a = 0;
  int h = 0;
  for (int w = 0; w < T.G; ++w) {
    a += lo[32 * w + T.lane];
    h += S.redh[32 * w + T.lane];
  }
  if (T.lane < k + 2) {
    R.lo[slot * (k + 2) + T.lane] = a;
    R.hi[slot * (k + 2) + T.lane] = h;
  }
}

// score_e += d_e - wsum_e / sume over the ring's first cnt ministeps (one warp):
// lane = 8 (e mod 4) + slot, the slots' terms added in a fixed tree, so the scores
// do not depend on the team size.
static __device__ __noinline__ void scores_flush(const ScoreRing R, const int *ecls,
                                                 const int *ety, const int *esd, double *sc,
                                                 int k, int lane, int cnt) {
  const int slot = lane & (kRing - 1);
  const int meta = slot < cnt ? R.meta[slot] : -1;
  const bool on = meta >= 0;
  const int sh = on ? meta >> 2 : 0, x = slot * (k + 2);
  const double dl = (meta & 1) ? 0.0 : ((meta & 2) ? -1.0 : 1.0);
  const double w = on ? count_sum(R, x) : 1.0, dw = on ? count_sum(R, x + 1) : 0.0;
  const double inv = __ddiv_rn(1.0, w);
  const int64_t stay = stay_weight(sh);
  auto term = [&](int e) -> double {
    if (!on || e >= k) return 0.0;
    const int cls = ecls[e] & 0xFF;
    const int64_t m = R.dst[slot * k + e];
    if (cls == FX_DELTA) return __dsub_rn(dl, __dmul_rn(dw, inv));
    if (cls == FX_UNI)   // a_ij = 0: the magnitude itself
      return __dmul_rn(__longlong_as_double(m), __dsub_rn(dl, __dmul_rn(dw, inv)));
    if (cls == FX_CNT)
      return __dsub_rn(__dmul_rn(dl, (double)m), __dmul_rn(count_sum(R, x + 2 + e), inv));
    if (cls != FX_REAL) return 0.0;
    const double back = pow2(-esd[e]);
    const double mean = __dmul_rn(__dmul_rn(sum_value(R, x, 2 + e, true, ety[e], stay), inv),
                                  __dmul_rn(pow2(58), back));
    // (a magnitude of 0 marks one that the type rules out)
    const double ds =
        m ? __dmul_rn(__dmul_rn(dl, (double)(int64_t)((uint64_t)m + kMinus62)), back) : 0.0;
    return __dsub_rn(ds, mean);
  };
  for (int e0 = 0; e0 < k; e0 += 8) {   // two effects at once: their chains overlap
    const int e = e0 + (lane >> 3);
    double c = term(e), c4 = term(e + 4);
#pragma unroll
    for (int o = 1; o < kRing; o <<= 1) {
      c = __dadd_rn(c, __shfl_xor_sync(kFull, c, o));
      c4 = __dadd_rn(c4, __shfl_xor_sync(kFull, c4, o));
    }
    if (slot == 0 && e < k) sc[e] = __dadd_rn(sc[e], c);
    if (slot == 0 && e + 4 < k) sc[e + 4] = __dadd_rn(sc[e + 4], c4);
  }
}
__device__ __forceinline__ void scores_flush(const Team &T, const Slice &S, int k, int cnt) {
  // not the first warp, whose lanes toggle the tie meanwhile
  if (T.warp == T.G - 1) scores_flush(ring_of(S, k), S.ecls, S.ety, S.esd, S.sc, k, T.lane, cnt);
}

constexpr int kLn2 = 11356;   // ln2 at scale 2^-14
// A predictor this many ln2 (11.8) below sh ln2 has a weight of fewer than 28 bits,
// whose rounding may exceed 2^-28 of it, a sixteenth of a float32's. From sh = 18 on
// that is the "no change" alter's, and the sums are formed in float64.
constexpr int kMaxShift = 17;
// Largest scaling that a ministep hands on, and the ministeps after which it drops by one.
constexpr int kKeepShift = 8, kShiftLife = 32;

// Whether a sum of the ring's slot may have lost a float32's precision to weights of
// few bits: it is below 2^34 units of the grid (of a real statistic as large as its
// bound 2^38), where hundreds of weights' roundings stay below 2^-29 of it; or it is 0
// and a weight was rounded to 0 (zeros). One warp.
static __device__ __noinline__ bool sums_short(const ScoreRing R, const int *ecls, const int *ety,
                                               int k, int slot, int sh, int lane, bool zeros) {
  if (lane >= k + 2) return false;
  const int x = slot * (k + 2), e = lane - 2, cls = e < 0 ? (int)FX_CNT : ecls[e] & 0xFF;
  if (cls < FX_CNT) return false;
  const double v = fabs(sum_value(R, x, lane, cls == FX_REAL, e < 0 ? 0 : ety[e], stay_weight(sh)));
  return v == 0.0 ? zeros : v < (cls == FX_REAL ? 274877906944.0 : 17179869184.0);
}

// Largest f (scale 2^-14) for which no lane's sums can leave 63 bits: with nb
// blocks of 32 alters a lane adds at most nb products w |d| at scale 2^44 (real
// statistics: w 2^50 at most), so w mb nb <= 2^17 keeps them below 2^61, mb
// being
// the largest count or degree that the ministep can meet (at least 16).
__device__ __forceinline__ int step_guard(const DevProblem &P, const Slice &S, const StepCtx &X) {
  const int nb = (P.n + 31) >> 5;
  int mb = max(16, max(2 * X.od_i + 2, X.id_i + 1));
  mb = max(mb, S.misc[10] + 1);
  // out-degrees of every network (cross effects count another network's ties)
  for (int w = 0; w < X.net.D; ++w) mb = max(mb, X.net.misc[w * X.net.misc_stride + 11] + 1);
  const int lg = 17 - (32 - __clz(mb * nb - 1));   // floor(log2(2^17 / (mb nb)))
  return lg * kLn2;
}

// Per-thread scratch of one alter's change statistics in the pass over the
// alters: the model's k in the specialised build, the capacity otherwise.
#if defined(CUSNA_JIT_K)
constexpr int kScratchK = CUSNA_JIT_K;
#else
constexpr int kScratchK = kMaxEff;
#endif

// Actor i's words of the out-row, in-row and permitted row, 32 at a time: lane l
// holds word first + l. The pass broadcasts a block's words by shuffles: three loads
// for 32 blocks, issued before the ministep's other work, in place of three per
// block, two of them global (the permitted row, and the in-row where the columns are
// in global scratch). Forward simulation n = 200, 4096 chains: 64.9 -> 61.1 ms;
// co-evolution n = 1000: 156 -> 137 ms.
struct RowWords {
  uint32_t out, in, ok;
  int first;
};
__device__ __forceinline__ RowWords row_words(const DevProblem &P, const Slice &S, int n, int W,
                                              int i, int first, int lane) {
  RowWords r{0u, 0u, 0u, first};
  const int w = first + lane;
  if (w < W) {
    r.out = S.rows[w * n + i];
    r.in = S.cols[w * n + i];
    r.ok = P.permr[w * n + i];
  }
  return r;
}

// The pass over the alters of one network ministep (see net_choice): per alter
// the magnitudes and the predictor, the float32 Gumbel key with its error bound
// (into *best and S.gbuf), the permitted-alter bits (S.okbits) and, with sums,
// the weight exp(f_j) 2^-sh and its products, whose warp sums end in S.red and
// S.redh. Returns the lane's largest predictor (scale 2^-14), and in fmin its
// smallest. Block b of 32 alters belongs to warp b mod G.
template <bool MULTI, bool VALID, int V>
__device__ __forceinline__ int alter_pass(const Team &T, const DevProblem &P, const Slice &S,
                                          const StepCtx &X, long long ms, uint32_t chain,
                                          KeyTop &best, int &fmin, bool sums, int sh, int net,
                                          RowWords words) {
  const int n = prob_n(P), k = prob_k(P), i = X.i;
  (void)net;
  const int nb = (n + 31) >> 5;
#ifdef CUSNA_JIT_K
  constexpr int KS = CUSNA_JIT_K;
#else
  const int KS = k;
#endif
  uint64_t acc[V];
#pragma unroll
  for (int q = 0; q < V; ++q) acc[q] = 0;
  int fmax = 0;
  fmin = 0;
  const bool full = P.maxdeg > 0 && X.od_i >= P.maxdeg;   // no new tie
  const uint32_t k0 = P.k0, k1 = P.k1;
#pragma unroll 1
  for (int b = T.warp; b < nb; b += T.G) {
    const int jl = (b << 5) + T.lane, j = jl < n ? jl : n - 1;
    if ((b & ~31) != words.first)   // n > 1024: the next 32 blocks' words
      words = row_words(P, S, n, prob_w(P), i, b & ~31, T.lane);
    const int aij = (__shfl_sync(kFull, words.out, b & 31) >> T.lane) & 1;
    const int aji = (__shfl_sync(kFull, words.in, b & 31) >> T.lane) & 1;
    const uint32_t permitted = (__shfl_sync(kFull, words.ok, b & 31) >> T.lane) & 1u;
    const bool stay = j == i;
    const bool ok = jl < n && (stay || (permitted && !(full && aij == 0)));
    const float gum = gumbel_est(alter_word<VALID>(P, S, ms, chain, j, k0, k1));
    uint64_t v[kScratchK];
#if defined(CUSNA_JIT_SPEC)
    int64_t f = jit_change_fixed(P, S, X, j, aij, aji, v);
#elif defined(CUSNA_JIT_MULTI)
    int64_t f = jit_change_fixed(net, P, S, X, j, aij, aji, v);
#else
    int64_t f = change_fixed<MULTI>(P, S, X, j, aij, aji, v);
#endif
    f = stay ? 0 : signed_fx((uint64_t)f, aij);
    const int fh = (int)(f >> 32);
    // float32 rounding of f 2^-46
    const float f32 = fmaf((float)fh, 6.103515625e-5f, __fmul_rn((float)(uint32_t)f, 1.4210854715202004e-14f));
    const float gk = __fsub_rn(f32, gum);
    const float E = fmaf(fabsf(f32), 3.6e-7f, 3e-5f);
    if (ok) {
      fmax = max(fmax, fh);
      fmin = min(fmin, fh);
      keytop_add(best, gk, E, j);
    }
    if (jl < n) S.gbuf[j] = ok ? __fadd_rn(gk, E) : -INFINITY;
    const uint32_t okb = __ballot_sync(kFull, ok);
    if (T.lane == 0) S.okbits[b] = okb;
    if (sums) {
      uint64_t W = exp_fx(f, sh, S.etab);
      if (!ok) W = 0;
      if (stay) {
        acc[0] += W;
      } else {
#if defined(CUSNA_JIT_SPEC)
        jit_sums_add(acc, W, aij, v);
#elif defined(CUSNA_JIT_MULTI)
        jit_sums_add(net, acc, W, aij, v);
#else
        sums_add<V>(S, KS, acc, W, aij, v);
#endif
      }
    }
  }
  if (sums) {
    int64_t lo;
    int hi;
    sums_reduce<V>(acc, T.lane, lo, hi);
    reinterpret_cast<int64_t *>(S.red)[32 * T.warp + T.lane] = lo;
    S.redh[32 * T.warp + T.lane] = hi;
  }
  return fmax;
}

// Every permitted alter a candidate for the float64 keys: a ministep of a chain
// outside the fixed-point range. (The functions of the rare paths take the slice
// by value: a reference would keep it in memory, and the hot path's shared-memory
// pointers with it.)
static __device__ __noinline__ void mark_all(const Team T, const DevProblem &P, const Slice S,
                                             const StepCtx X) {
  const int n = P.n, i = X.i;
  const bool full = P.maxdeg > 0 && X.od_i >= P.maxdeg;
  for (int b = T.warp; b < ((n + 31) >> 5); b += T.G) {
    const int j = (b << 5) + T.lane;
    const bool ok = j < n && (j == i || (bit_of(P.permr, n, i, j) &&
                                         !(full && bit_of(S.rows, n, i, j) == 0)));
    if (j < n) S.gbuf[j] = ok ? INFINITY : -INFINITY;
    const uint32_t okb = __ballot_sync(kFull, ok);
    if (T.lane == 0) S.okbits[b] = okb;
  }
  T.sync();
}

// The choice by exact float64 keys among the permitted alters whose upper bound
// is not below lb (the reference's f_j - log(-log u_j), ties to the smaller j).
template <bool MULTI, bool VALID>
static __device__ __noinline__ int choice_float64(const Team T, const DevProblem &P, const Slice S,
                                                  const StepCtx X, long long ms, uint32_t chain,
                                                  float lb, double *d, int net) {
  const int n = P.n, i = X.i;
  long long bk = dkey(-1e300);
  int bj = 0x7FFFFFFF;
  for (int j = T.tl; j < n; j += T.L) {
    const bool okj = (S.okbits[j >> 5] >> (j & 31)) & 1u;
    if (okj && !(S.gbuf[j] < lb)) {
      const double f = j != i ? f64_of<MULTI>(P, S, X, j, d, net) : 0.0;
      const double g = __dsub_rn(f, log(-log(unif01(alter_word<VALID>(P, S, ms, chain, j, P.k0, P.k1)))));
      if (is_nan64(g)) continue;
      const long long kg = dkey(g);
      if (kg > bk || (kg == bk && j < bj)) { bk = kg; bj = j; }
    }
  }
  return team_argmax(T, bk, bj, S.red + 32 * T.G + 32);
}

// The chain's scores go through the ring.
__device__ __forceinline__ bool ring_scores(const DevProblem &P, const Slice &S) {
  return (P.flags & (F_NO_SCORES | F_LSE64)) == 0 && S.misc[15] != 0;
}
// After ministep slot's choice and a team barrier: a full ring into the scores.
__device__ __forceinline__ void score_slot(const Team &T, const DevProblem &P, const Slice &S,
                                           int slot) {
  if (slot == kRing - 1 && ring_scores(P, S)) scores_flush(T, S, prob_k(P), kRing);
}

// One network ministep of focal actor i on the network of slice S, up to the
// choice: the pass over the alters and the certified or exact float64 choice.
// Returns j*. The score sums and the chosen alter's magnitudes go to slot of the
// ring, which the caller flushes after a team barrier (score_slot). d (float64)
// is per-thread scratch of k values.
// MULTI: the network is one of a multi-network problem's. nb0 locates the state
// of every network (of the one network).
// VALID: validation mode (caller-supplied words in place of Philox).
template <bool MULTI, bool VALID = false>
__device__ __forceinline__ int net_choice(const Team &T, const DevProblem &P, const Slice &S,
                                          int i, long long ms, uint32_t chain, double *d,
                                          const NetBase *nb0, int slot, int &keep, int net = 0) {
  const int n = prob_n(P), W = prob_w(P), k = prob_k(P), L = T.L, fl = P.flags;
  (void)net;
  const RowWords words = row_words(P, S, n, W, i, 0, T.lane);
  StepCtx X;
  X.i = i;
  X.od_i = S.outdeg[i];
  X.id_i = S.indeg[i];
  X.rdeg_i = 0;
  if (fl & F_NEED_RDEG)
    for (int w = 0; w < W; ++w) X.rdeg_i += __popc(S.rows[w * n + i] & S.cols[w * n + i]);
  X.zvi = (fl & F_HAS_Z) ? __dsub_rn((double)S.z[i], P.zbar) : 0.0;
  X.net = *nb0;
  X.tabq = P.tabq;
  step_helpers(T, P, S, X);
  X.f0 = S.fx[0];
  const bool ranged = S.fx[1] != 0;
  if (fl & F_HAS_STEP) {
    step_values(T, P, S, X);
    T.sync();
    if (ranged)
      for (int e = 0; e < k; ++e)
        if ((S.ecls[e] & 0xFF) == FX_UNI)
          X.f0 = (int64_t)((uint64_t)X.f0 +
                           (uint64_t)term_fx(S.thq[e], S.ecls[e], S.stepq[4 * e]));
  }

  // ---- one pass over the alters (alter_pass) -------------------------------
  // The key's error: f32 is within 2 2^-24 |f32| of the fixed-point predictor,
  // itself within 3k 2^-46 + 2^-50 (the tables) of the float64 f_j; gumbel_est
  // is within kGumbelErr; the subtraction rounds by 2^-24 (|f32| + 23). All of
  // it is below E_j = 3.6e-7 |f32| + 3e-5 (kGumbelErr + 1.4e-6 + the rest, twice).
  // gbuf[j] keeps the upper bound g_j + E_j. When a predictor exceeds the room
  // that the sums have (step_guard), the pass is repeated with every weight
  // scaled by 2^-sh, sh from the largest predictor (so from the alters alone). The
  // next ministep of the chain begins with that sh (keep: up to kKeepShift, less by
  // one every kShiftLife): in dense networks every other actor needs one, and 1,024
  // chains of n ~ U{20..400} at densities up to 0.1 took 36.7 ms with every ministep
  // beginning at 0, 33.6 so.
  // Where an alter's weight then has few bits and a sum is short of them
  // (sums_short), the ministep's sums are formed in float64: an effect whose
  // statistics are all at improbable alters has a score of its own size, and a
  // float32 ulp of that. (The fixed grid alone was 5e-6 of such a score off at
  // f = -20, and all of it from f = -31 on.)
  // Without requested scores (F_NO_SCORES) no sums are formed.
  const bool want_sums = (fl & F_NO_SCORES) == 0;
  const bool fast_sums = want_sums && (fl & F_LSE64) == 0 && ranged;
  KeyTop top{-INFINITY, 0.f, INFINITY, 0x7FFFFFFF};
  float lb = -INFINITY;
  int sh = fast_sums ? keep : 0, fn = 0;
  bool few = false, ring = false;
  if (ranged) {
    const int room = fast_sums ? step_guard(P, S, X) : 0x7FFFFFFF;
    for (;;) {
      KeyTop best{-INFINITY, 0.f, -INFINITY, 0x7FFFFFFF};
      int fm;
#ifdef CUSNA_FX_V
      fm = alter_pass<MULTI, VALID, CUSNA_FX_V>(T, P, S, X, ms, chain, best, fn, fast_sums, sh, net,
                                                words);
#else
      if (k + 2 <= 8)
        fm = alter_pass<MULTI, VALID, 8>(T, P, S, X, ms, chain, best, fn, fast_sums, sh, net, words);
      else if (k + 2 <= 16)
        fm = alter_pass<MULTI, VALID, 16>(T, P, S, X, ms, chain, best, fn, fast_sums, sh, net, words);
      else
        fm = alter_pass<MULTI, VALID, 26>(T, P, S, X, ms, chain, best, fn, fast_sums, sh, net, words);
#endif
      top = warp_keytop(best, T.lane);
      fm = __reduce_max_sync(kFull, fm);
      few = __any_sync(kFull, fn < (sh - kMaxShift) * kLn2);
      if (T.G > 1) {
        float *rb = reinterpret_cast<float *>(S.red + 32 * T.G + 32);   // 4 words per warp
        int *ri = reinterpret_cast<int *>(rb);
        if (T.lane == 0) {
          rb[4 * T.warp] = top.b1;
          rb[4 * T.warp + 1] = top.e1;
          rb[4 * T.warp + 2] = top.ub2;
          ri[4 * T.warp + 3] = top.j1;
          S.rfm[T.warp] = 2 * fm + (int)few;   // fm >= 0, the "no change" alter's
        }
        T.sync();
        top = KeyTop{rb[0], rb[1], rb[2], ri[3]};
        fm = S.rfm[0];
        int any = fm;
        for (int w = 1; w < T.G; ++w) {
          keytop_merge(top, KeyTop{rb[4 * w], rb[4 * w + 1], rb[4 * w + 2], ri[4 * w + 3]});
          fm = max(fm, S.rfm[w]);
          any |= S.rfm[w];
        }
        fm >>= 1;
        few = any & 1;
      } else {
        __syncwarp();
      }
      if (__builtin_expect(fm <= room + sh * kLn2 || !fast_sums, 1)) break;
      // the smallest scaling for which the largest predictor fits
      sh = (fm - room + kLn2 - 1) / kLn2;
      if (sh > kMaxShift) break;
      T.sync();   // every warp has read the first pass's scratch
    }
    ring = fast_sums && sh <= kMaxShift;
    keep = max(min(sh, kKeepShift) - (int)(((int)ms & (kShiftLife - 1)) == 0), 0);
    if (__builtin_expect(ring && few, 0)) {
      const bool z = __any_sync(kFull, fn < (sh - kWBits + 1) * kLn2);
      T.sync();   // every warp has read rfm
      if (T.lane == 0) S.rfm[T.warp] = z;
      T.sync();
      if (T.warp == 0) {
        int zeros = 0;
        for (int w = 0; w < T.G; ++w) zeros |= S.rfm[w];
        sums_combine(T, S, ring_of(S, k), k, slot);
        __syncwarp();
        const bool s = __any_sync(kFull, sums_short(ring_of(S, k), S.ecls, S.ety, k, slot, sh, T.lane,
                                                    zeros != 0));
        if (T.lane == 0) S.rfm[0] = s;
      }
      T.sync();
      ring = S.rfm[0] == 0;
    }
    lb = __fsub_rn(top.b1, top.e1);
  } else {
    mark_all(T, P, S, X);
  }

  // ---- the chosen alter ---------------------------------------------------
  // The float32 keys decide when the best key's lower bound exceeds every
  // other alter's upper bound; otherwise the exact float64 keys of the permitted
  // alters that reach it decide. The "no change" alter always has a finite key,
  // so a choice always exists.
  int jstar = lb > top.ub2 ? top.j1
                           : choice_float64<MULTI, VALID>(T, P, S, X, ms, chain, lb, d, net);
  // never an index outside the network, whatever the inputs
  if ((unsigned)jstar >= (unsigned)n) jstar = i;

  // the score sums into the ring by a warp other than the chosen alter's owner,
  // which meanwhile forms the chosen alter's magnitudes; on the float64 path, the
  // scores by the whole team
  if (want_sums && !ring) {
    if (T.tl == 0) ring_of(S, k).meta[slot] = -1;
#ifdef CUSNA_JIT_K
    lse_float64<MULTI, CUSNA_JIT_K + 1>(T, P, S, X, d, net, jstar);
#else
    if (k + 1 <= 8) lse_float64<MULTI, 8>(T, P, S, X, d, net, jstar);
    else if (k + 1 <= 16) lse_float64<MULTI, 16>(T, P, S, X, d, net, jstar);
    else lse_float64<MULTI, 32>(T, P, S, X, d, net, jstar);
#endif
  } else if (ring) {
    const ScoreRing R = ring_of(S, k);
    const int owner = jstar & (L - 1);   // L and G are powers of two
    if (T.warp == (((owner >> 5) + 1) & (T.G - 1))) sums_combine(T, S, R, k, slot);
    if (T.tl == owner) {
      const int aij = bit_of(S.rows, n, i, jstar), aji = bit_of(S.cols, n, i, jstar);
      uint64_t *v = reinterpret_cast<uint64_t *>(R.dst) + slot * k;
      R.meta[slot] = 4 * sh + 2 * aij + (jstar == i ? 1 : 0);
      if (jstar == i) {
        for (int e = 0; e < k; ++e) v[e] = 0;
      } else {
#if defined(CUSNA_JIT_SPEC)
        jit_change_fixed(P, S, X, jstar, aij, aji, v);
#elif defined(CUSNA_JIT_MULTI)
        jit_change_fixed(net, P, S, X, jstar, aij, aji, v);
#else
        change_fixed<MULTI>(P, S, X, jstar, aij, aji, v);
#endif
      }
      if (fl & F_HAS_STEP)
        for (int e = 0; e < k; ++e)
          if ((S.ecls[e] & 0xFF) == FX_UNI) v[e] = (uint64_t)__double_as_longlong(S.stepd[4 * e]);
    }
  }
  return jstar;
}

// Toggles the tie i -> j (dl = +-1; and j -> i, symmetric): the bits by lanes 0
// and 1, the degrees and their largest values by lanes 2 and 3 (4..7: the other
// direction), each access of all of them at once. The two directions write
// different words, except the largest degrees.
__device__ __forceinline__ void toggle_tie(const Team &T, const Slice &S, int n, int i, int j,
                                           int dl, int symflag) {
  if (T.tl >= (symflag ? 8 : 4)) return;
  const int u = T.tl & 4 ? j : i, v = T.tl & 4 ? i : j;
  if ((T.tl & 2) == 0) {
    uint32_t *w = T.tl & 1 ? S.cols + (u >> 5) * n + v : S.rows + (v >> 5) * n + u;
    *w ^= 1u << ((T.tl & 1 ? u : v) & 31);
  } else {
    short *d = T.tl & 1 ? S.outdeg + u : S.indeg + v;
    const int x = *d + dl;
    *d = (short)x;
    atomicMax(S.misc + 10 + (T.tl & 1), x);
  }
}

// Validation trace record of ministep ms (validation mode only): (step,
// focal actor, choice, change of the distance); the choice is the chosen alter
// of a network ministep, or -(d + 2) for a behaviour step d.
template <bool VALID>
__device__ __forceinline__ void trace_put(const DevProblem &P, int c, long long ms, int actor,
                                          int choice, long long delta) {
  if (!VALID || !P.trace || ms >= P.trace_cap) return;
  int *t = P.trace + ((size_t)c * P.trace_cap + (size_t)ms) * 4;
  t[0] = (int)ms;
  t[1] = actor;
  t[2] = choice;
  t[3] = (int)delta;
}

// One chain: the ministep loop and the chain's outputs.
template <bool VALID>
static __device__ void run_chain(const Team &T, const DevProblem &P, const Slice &S, int c) {
  const int n = prob_n(P), k = prob_k(P);
  const uint32_t chain = P.chain_offset + (uint32_t)c;
  chain_init(T, P, S, c);

  const double lam = (double)P.lam[c * P.prow];
  const double lamb = P.lamb ? (double)P.lamb[c * P.prow] : 0.0;
  // the reference's constant-rate expressions (src/libcusna_saom_cpu.cpp:195,197)
  const double den = __dmul_rn((double)P.nact, __dadd_rn(lam, lamb));
  const double pnet = __ddiv_rn(lam, __dadd_rn(lam, lamb));
  long long dist = 0, bdist = 0, ms = 0, msb = 0;
  double t = 0.0, rho = 0.0, tnext = 0.0;
  bool over = false;   // tnext ends an unconditional period
  int keep = 0;        // the score sums' scaling to begin with (net_choice)
  double d[kMaxEff];
  const NetBase nb{S.rows, S.cols, S.cm, 0, 0, 0, S.misc, 0, 1};

  for (;;) {
    int i;
    bool is_net;
    uint32_t r3;
    if (P.nrate > 0) {
      uint32_t rr[4];
      step_words<VALID>(P, S, ms, chain, rr);
      if (((int)ms & (kCapEvery - 1)) == 0 && T.tl == 0) cap_check(S);
      i = rate_draw(T, P, S, rr, lam, t, rho);
      if (i < 0) break;
      is_net = true;
      r3 = rr[3];
    } else {
      // constant rate (:195-199). The draws of 32 ministeps are formed at
      // once, one per lane of warp 0 (they depend only on the counters), and
      // the time is accumulated in order, so every value equals the reference's.
      const int slot = (int)(ms & 31);
      if (slot == 0) {
        if (T.warp == 0) {
          uint32_t rr[4];
          step_words<VALID>(P, S, ms + T.lane, chain, rr);
          S.rtau[T.lane] = __ddiv_rn(-log(unif01(rr[0])), den);
          S.rnet[T.lane] = (P.kb == 0 || unif01(rr[1]) < pnet) ? 1 : 0;
          long long idx = (long long)__dmul_rn(unif01(rr[2]), (double)P.nact);
          if (idx >= P.nact) idx = P.nact - 1;
          S.rfocal[T.lane] = P.act[idx];
          S.rr3[T.lane] = rr[3];
          if (T.lane == 0) cap_check(S);
        }
        T.sync();
        tnext = __dadd_rn(t, S.rtau[0]);
        over = !P.cond && tnext > 1.0;
      }
      // the time after the following ministep is formed while this one runs
      t = tnext;
      if (over) break;
      if (slot < 31) {
        tnext = __dadd_rn(t, S.rtau[slot + 1]);
        over = !P.cond && tnext > 1.0;
      }
      is_net = S.rnet[slot] != 0;
      i = S.rfocal[slot];
      r3 = S.rr3[slot];
    }

    if (!is_net) {
      if (T.warp == 0) {
        const long long bd0 = bdist;
        const int dz = beh_step(T, P, S, i, r3, &bdist);
        if (T.lane == 0) trace_put<VALID>(P, c, ms, i, -(dz + 2), bdist - bd0);
      }
      T.sync();
      ++msb;
      ++ms;
      if (P.cond && dist >= P.target_dist) break;
      if (ms >= kMaxSteps) break;
      continue;
    }

    const int rslot = (int)(ms - msb) & (kRing - 1);
    const int jstar = net_choice<false, VALID>(T, P, S, i, ms, chain, d, &nb, rslot, keep);
    const int aij_star = bit_of(S.rows, n, i, jstar);
    T.sync();
    score_slot(T, P, S, rslot);
    const long long dist0 = dist;
    ++ms;
    if (jstar != i) {
      const int j = jstar;
      const long long chg = P.symflag ? 2 : 1;
      // (the distance's words are used after the toggle, off its path)
      const uint32_t kd = P.kdistr[(j >> 5) * n + i], x0 = P.x0r[(j >> 5) * n + i];
      if (P.cnt.mask)
        counts_toggle(T, P, nb, i, j, 1 - 2 * aij_star);
      toggle_tie(T, S, n, i, j, 1 - 2 * aij_star, P.symflag);
      if ((kd >> (j & 31)) & 1u)
        dist += (uint32_t)aij_star == ((x0 >> (j & 31)) & 1u) ? chg : -chg;
    }
    if (T.tl == 0) trace_put<VALID>(P, c, ms - 1, i, jstar, dist - dist0);
    if (P.nrate > 0) T.sync();   // the degrees below are the toggled ones (toggle_tie's lanes)
    if (P.nrate > 0 && T.tl == 0) {
      for (int q = 0; q < P.nrate; ++q) {
        const int rk = S.rkind[q];
        const double u = rk == 0 ? P.ru[(size_t)q * n + i]
                                 : (rk == 1 ? (double)S.outdeg[i] : (double)S.indeg[i]);
        S.rsc[q] = __dadd_rn(S.rsc[q], u);
      }
    }
    T.sync();
    if (P.cond && dist >= P.target_dist) break;
    if (ms >= kMaxSteps) break;
  }

  T.sync();
  if (((ms - msb) & (kRing - 1)) && ring_scores(P, S))
    scores_flush(T, S, k, (int)(ms - msb) & (kRing - 1));
  chain_finish(T, P, S, c, dist, bdist, ms, msb, t, rho, lam, lamb);
}

}  // namespace cusna
