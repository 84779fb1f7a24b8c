// saom_stats.cuh -- evaluation statistics of a network held in a team slice,
// and the end-of-chain outputs.
//
// Restates src/libcusna_saom_cpu.cpp:608-689 (cusna_network_stats) on
// word-major bitsets. Integer-valued statistics (tie counts, two-path sums,
// squared degrees, 0/0.5/1 indicator sums) are exact in any order and are
// summed by all lanes. Every other statistic is a float64 sum whose rounding
// depends on the order and is added in the reference's order (actors ascending, or
// ties or pairs in row-major order), giving identical bits: the lanes form 32
// terms of every such statistic at a time in shared memory, then one lane per
// statistic adds its own, so the serial chains of all statistics run side by side
// in one warp. A zero term changes no sum (a sum starts at +0 and is never -0)
// and is left out: most pairs' gwdsp weights are zero.
// This bounds the kernel: a dependent FP64 addition costs tens of cycles and an FP64
// instruction of a warp 16 issue cycles, whether 1 lane or 32 are active.
#pragma once
#include "saom_kernel.cuh"

namespace cusna {

// src/libcusna_saom_cpu.cpp:608-616
__device__ __forceinline__ double deg_term(int t, double pm, double cur, double start) {
  if (t == 8 || t == 9) {
    if (pm >= 1.0) return t == 9 ? sqrt(cur) : cur;
    return pm == 0.0 ? start : __dadd_rn(cur, start);
  }
  if (pm >= 1.0) return t == 15 ? sqrt(cur) : cur;
  const double s = pm == 0.0 ? start : __dadd_rn(cur, start);
  return t == 15 ? sqrt(s) : s;
}

struct StatDesc {
  const double *vmat, *vb, *wtab, *p1, *p2;
  const uint8_t *vmiss;
  const int *dyn, *od0, *id0, *type_ids;
  int n, W, k, symflag;
};

// The order-dependent statistics' kinds: 1 per actor, 2 per tie, 3 per pair.
__device__ __forceinline__ int stat_order(int t) {
  switch (t) {
    case 7: case 8: case 9: case 10: case 11: case 14: case 15: case 17: case 18: return 1;
    case 12: case 21: case 24: case 25: case 26: case 27: case 28: return 2;
    case 29: case 30: return 3;
    default: return 0;
  }
}

// Term of statistic e (type t) for actor j (order 1), or for the tie or pair (i, j).
// Returns 0 where the reference adds none.
template <class DegT>
__device__ __forceinline__ double stat_term(const StatDesc &D, const uint32_t *R,
                                            const uint32_t *Cc, const DegT *outdeg,
                                            const DegT *indeg, int e, int t, int i, int j) {
  const int n = D.n, W = D.W;
  const double pm = D.p1 ? D.p1[e] : 0.0;
  const bool dy = D.dyn && D.dyn[e];
  auto V = [&](int x) -> double {
    return dy ? (D.vb ? D.vb[x] : 0.0) : (D.vmat ? D.vmat[(size_t)e * n + x] : 0.0);
  };
  auto MISS = [&](int x) -> bool { return D.vmiss && D.vmiss[(size_t)e * n + x]; };
  switch (t) {
    case 7: case 17: return pow((double)(t == 7 ? indeg[j] : outdeg[j]), 1.5);
    case 8: case 9:
      return __dmul_rn((double)indeg[j], deg_term(t, pm, (double)outdeg[j], D.od0 ? (double)D.od0[j] : 0.0));
    case 14: case 15:
      return __dmul_rn((double)outdeg[j], deg_term(t, pm, (double)indeg[j], D.id0 ? (double)D.id0[j] : 0.0));
    case 18: return fmin((double)outdeg[j], pm);
    case 10: return MISS(j) ? 0.0 : __dmul_rn((double)outdeg[j], V(j));
    case 11: return MISS(j) ? 0.0 : __dmul_rn((double)indeg[j], V(j));
    case 12: case 21: case 25: {
      if (MISS(i) || MISS(j)) return 0.0;
      if (t == 12) {
        const double q2 = D.p2 ? D.p2[e] : 0.0;
        return __dsub_rn(__dsub_rn(1.0, __dmul_rn(fabs(__dsub_rn(V(i), V(j))), pm)), q2);
      }
      return t == 21 ? __dmul_rn(V(i), V(j)) : __dadd_rn(V(i), V(j));
    }
    default: {
      const double *wr = D.wtab + (size_t)e * (n + 1);
      if (t == 24 || t == 29) return wr[pc2(R, i, Cc, j, n, W)];   // (a@a)_ij
      if (t == 26 || t == 30) return wr[pc2(R, i, R, j, n, W)];    // (a@a^T)_ij
      if (t == 27) return wr[pc2(Cc, i, Cc, j, n, W)];             // (a^T@a)_ij
      return wr[pc2(Cc, i, R, j, n, W)];                           // (a^T@a^T)_ij
    }
  }
}

// The order-dependent statistics, up to `rows` of them at a time: statistic
// eid[q]'s terms in buf[33 q + x] (33: the adding lanes then read different banks),
// their number in cnt[q]. red holds eid and cnt (32 bytes each) and 33 rows doubles.
// Actors and pairs come by words of 32; ties by their rank, 32 at a time (a word of
// a sparse row holds less than one).
constexpr int kStatRow = 33;
__host__ __device__ inline size_t stat_scratch(int rows) { return 8 + (size_t)kStatRow * rows; }
template <class DegT>
static __device__ __noinline__ void ordered_stats(const Team T, const StatDesc &D,
                                                  const uint32_t *R, const uint32_t *Cc,
                                                  const DegT *outdeg, const DegT *indeg,
                                                  double *red, int rows, double *out) {
  const int n = D.n, W = D.W, k = D.k;
  unsigned char *eid = reinterpret_cast<unsigned char *>(red), *cnt = eid + 32;
  double *buf = red + 8;
  if (rows > 32) rows = 32;
  for (int kind = 1; kind <= 3; ++kind) {
    int e0 = 0;
    while (e0 < k) {
      T.sync();   // the scratch is free
      // the next group of statistics of this kind
      int have = 0;
      for (; e0 < k && have < rows; ++e0)
        if (stat_order(D.type_ids[e0]) == kind) {
          if (T.tl == 0) eid[have] = (unsigned char)e0;
          ++have;
        }
      if (have == 0) break;
      T.sync();
      double acc = 0.0;
      // the first tie (by rank) of a batch, and the row that holds it with the
      // number of ties before that row
      int start = 0, row = 0, before = 0;
      for (int i = 0, w = 0;;) {
        int a = i, j;
        bool on, more;
        if (kind == 2) {
          int r = row, c = before, x = start + T.lane;
          while (r < n && c + (int)outdeg[r] <= x) c += (int)outdeg[r++];
          on = r < n;
          j = 0;
          if (on) {
            int left = x - c, v = 0;
            uint32_t m = R[r];
            while (left >= __popc(m)) {
              left -= __popc(m);
              m = R[(++v) * n + r];
            }
            while (left-- > 0) m &= m - 1;
            j = (v << 5) + __ffs(m) - 1;
          }
          a = r;
          row = __shfl_sync(kFull, r, 31);
          before = __shfl_sync(kFull, c, 31);
          start += 32;
          more = row < n;
          if (!__any_sync(kFull, on)) break;
        } else {
          j = (w << 5) + T.lane;
          on = j < n && !(kind == 3 && j == i);
          more = true;
        }
        for (int q = T.warp; q < have; q += T.G) {
          const int e = eid[q];
          const double term = on ? stat_term(D, R, Cc, outdeg, indeg, e, D.type_ids[e], a, j) : 0.0;
          const bool keep = term != 0.0;   // true for a NaN
          const uint32_t m = __ballot_sync(kFull, keep);
          if (keep) buf[kStatRow * q + __popc(m & ((1u << T.lane) - 1u))] = term;
          if (T.lane == 0) cnt[q] = (unsigned char)__popc(m);
        }
        T.sync();
        if (T.warp == 0 && T.lane < have) {
          const int c = cnt[T.lane];
          const double *b = buf + kStatRow * T.lane;
          for (int x = 0; x < c; x += 4) {   // x + 3 <= 31: within the row
            const double v0 = b[x], v1 = b[x + 1], v2 = b[x + 2], v3 = b[x + 3];
            acc = __dadd_rn(acc, v0);
            if (x + 1 < c) acc = __dadd_rn(acc, v1);
            if (x + 2 < c) acc = __dadd_rn(acc, v2);
            if (x + 3 < c) acc = __dadd_rn(acc, v3);
          }
        }
        T.sync();
        if (kind == 2) {
          if (!more) break;
        } else if (++w == W) {
          w = 0;
          if (kind == 1 || ++i == n) break;
        }
      }
      if (T.warp == 0 && T.lane < have) out[eid[T.lane]] = acc;
    }
  }
}

// Statistics of the network in (R, C) (word-major rows / in-rows) with degrees
// outdeg/indeg already filled. red: stat_scratch(rows) doubles of team scratch
// (at least 32 G).
template <class DegT>
__device__ inline void network_stats_team(const Team &T, const StatDesc &D, const uint32_t *R,
                                          const uint32_t *Cc, const DegT *outdeg,
                                          const DegT *indeg, double *red, int rows, double *out) {
  const int n = D.n, W = D.W, k = D.k;
  for (int e = 0; e < k; ++e) {
    const int t = D.type_ids[e];
    const double pm = D.p1 ? D.p1[e] : 0.0;
    const bool dy = D.dyn && D.dyn[e];
    auto V = [&](int x) -> double {
      return dy ? (D.vb ? D.vb[x] : 0.0) : (D.vmat ? D.vmat[(size_t)e * n + x] : 0.0);
    };
    auto MISS = [&](int x) -> bool { return D.vmiss && D.vmiss[(size_t)e * n + x]; };
    double acc = 0.0;
    bool integer = true;
    long long part = 0;
    switch (t) {
      case 0: case 1: case 2: case 3: case 23: case 5: case 6: case 4: case 16: case 19:
      case 13: case 20: case 31:
        // integer-valued (20 counts halves): all lanes, one row i per lane
        for (int i = T.tl; i < n; i += T.L) {
          long long s = 0;
          if (t == 0) s = outdeg[i];
          else if (t == 4) s = (long long)indeg[i] * indeg[i];
          else if (t == 16) s = (long long)outdeg[i] * outdeg[i];
          else if (t == 1 || t == 19) {
            int rd = 0;
            for (int w = 0; w < W; ++w) rd += __popc(R[w * n + i] & Cc[w * n + i]);
            s = t == 1 ? rd : (long long)outdeg[i] * rd;
          } else {
            for (int w = 0; w < W; ++w) {
              uint32_t m = R[w * n + i];
              if (t == 6) m &= Cc[w * n + i];
              while (m) {
                const int j = (w << 5) + __ffs(m) - 1;
                m &= m - 1;
                if (t == 2 || t == 23 || t == 5 || t == 6) {
                  const int aa = pc2(R, i, Cc, j, n, W);  // (a@a)_ij
                  s += (t == 5) ? (aa > 0) : aa;
                } else if (t == 3) {
                  s += pc2(R, j, Cc, i, n, W);            // tie i->j adds (a@a)_ji
                } else if (t == 13) {
                  if (!MISS(i) && !MISS(j)) s += fabs(V(i) - V(j)) < 1e-9 ? 1 : 0;
                } else if (t == 20) {  // twice the term: 0, 1 or 2
                  if (MISS(i) || MISS(j)) s += 1;
                  else {
                    const double dd = V(i) - V(j);
                    s += 2 * (dd > 1e-9 ? 1 : 0) + (fabs(dd) <= 1e-9 ? 1 : 0);
                  }
                } else if (t == 31) {
                  if (!MISS(j) && V(j) >= pm - 1e-12) s += 1;
                }
              }
            }
          }
          part += s;
        }
        part = team_sum_ll(T, part, red);
        acc = (double)part;
        if (t == 0 && D.symflag) acc = acc * 0.5;
        if (t == 3) acc = acc / 3.0;
        if (t == 23) acc = acc / 6.0;
        if (t == 20) acc = acc * 0.5;
        break;
      default:
        integer = false;
        break;
    }
    if (integer) {
      if (T.tl == 0) out[e] = acc;
    } else if (T.tl == 0 && stat_order(t) == 0) {
      out[e] = 0.0;   // 22, 32 and others: the reference reports 0
    }
  }
  ordered_stats(T, D, R, Cc, outdeg, indeg, red, rows, out);
}

// End of one chain (src/libcusna_saom_cpu.cpp:290-302 and :394-422).
__device__ void chain_finish(const Team &T, const DevProblem &P, const Slice &S, int c,
                             long long dist, long long bdist, long long ms, long long msb,
                             double t, double rho, double lam, double lamb);

}  // namespace cusna
