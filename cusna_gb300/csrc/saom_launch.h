// saom_launch.h -- launch wrappers shared by the kernels (saom_sim.cu) and the
// host code (saom_api.cu).
#pragma once
#include <nvtx3/nvToolsExt.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "saom_common.cuh"
#include "saom_kernel.cuh"
#include "libcusna.h"

namespace cusna {

struct StatDesc;

// Launch shape of the period kernel, chosen by the autotuner (saom_api.cu).
struct LaunchShape {
  int G;              // warps per chain
  int teams_per_cta;  // chains per CTA
  int ctas;           // grid size (persistent: ctas * teams_per_cta resident teams)
  bool cols_in_smem;  // in-rows in shared memory (else global scratch)
  bool rows_in_smem;  // out-rows in shared memory (else global scratch)
  SliceLayout lay;
};

// Global scratch of a launch, one piece per team (and network): the chain's
// in-rows and out-rows (cols_words each; null where the slice holds them) and
// its count matrices (counts_stride counts; null without).
struct Scratch {
  uint32_t *cols = nullptr, *rows = nullptr;
  uint16_t *counts = nullptr;
  size_t cols_words = 0, counts_stride = 0;
};

// The two-path counters of a model's effects and each effect's packed count
// function (cfn_pack): fn[e] and the counters it reads. multi: cross effects
// (types 36, 37) read network cross_src[e].
inline void plan_counters(const int *tid, int k, bool multi, const int *cross_src, CounterSet &C,
                          int *packed) {
  C.n = 0;
  C.mask = 0;
  C.ntask = 0;
  C.tp = C.tq = -1;
  auto add = [&](int list, int m1, int m2 = CM_NONE) -> int {
    for (int c = 0; c < C.n; ++c)
      if (C.list[c] == list && C.m1[c] == m1 && C.m2[c] == m2) return c;
    C.list[C.n] = (unsigned char)list;
    C.m1[C.n] = (unsigned char)m1;
    C.m2[C.n] = (unsigned char)m2;
    return C.n++;
  };
  for (int e = 0; e < k; ++e) {
    int &p = packed[e];
    p = cfn_pack(0);
    switch (tid[e]) {
      case 2: p = cfn_pack(2, add(CL_OUT, CM_ROWS, CM_COLS)); break;
      case 3: case 23: p = cfn_pack(3, add(CL_IN, CM_COLS)); break;
      case 5: {
        C.tp = add(CL_OUT, CM_ROWS);
        const int a = add(CL_TP0, CM_COLS), b = add(CL_TP1, CM_COLS);
        p = cfn_pack(5, a, b, C.tp);
        break;
      }
      case 6: {
        const int a = add(CL_OUT, CM_ROWS), b = add(CL_MUTUAL, CM_COLS);
        p = cfn_pack(6, a, b);
        break;
      }
      case 24: p = cfn_pack(8, add(CL_OUT, CM_ROWS)); break;
      case 26: p = cfn_pack(8, add(CL_OUT, CM_COLS)); break;
      case 27: p = cfn_pack(8, add(CL_IN, CM_ROWS)); break;
      case 28: p = cfn_pack(8, add(CL_IN, CM_COLS)); break;
      case 29: C.tp = add(CL_OUT, CM_ROWS); break;
      case 30: C.tq = add(CL_OUT, CM_COLS); break;
      case 36:
        if (multi) p = cfn_pack(36, add(CL_NET + cross_src[e], CM_NCOLS + cross_src[e]));
        break;
      case 37:
        if (multi) p = cfn_pack(37, add(CL_NET + cross_src[e], CM_ROWS));
        break;
      default: break;
    }
  }
}

// The updates of the count matrices when a tie toggles in network x: for the
// counters (masked) of network d = 0..D-1 that read x. A counter is the product
// C = L M of its set's relation L (i to h) and its relation M (h to j), so
// toggling L's tie (i, h) adds row h of M to row i of C, and toggling M's tie
// (h, j) adds column h of L to column j of C; both cannot meet off the diagonal.
inline void counter_tasks(const CounterSet *const *nets, int D, int x, CounterSet &out) {
  out.ntask = 0;
  for (int d = 0; d < D; ++d) {
    const CounterSet &C = *nets[d];
    for (int c = 0, rank = 0; c < C.n; ++c) {
      if (!((C.mask >> c) & 1u)) continue;
      const bool lin = C.list[c] == CL_IN;
      const int netL = C.list[c] >= CL_NET ? C.list[c] - CL_NET : d;
      for (int m : {(int)C.m1[c], (int)C.m2[c]}) {
        if (m == CM_NONE) continue;
        const bool mrows = m == CM_ROWS;
        const int netM = m >= CM_NCOLS ? m - CM_NCOLS : d;
        // L's tie: i = u, h = v (CL_IN: i = v, h = u); row h of M into row i
        if (netL == x) out.task[out.ntask++] = task_pack(!mrows, !lin, lin, false, rank, netM, d);
        // M's tie: h = u, j = v (its transpose: h = v, j = u); column h of L into column j
        if (netM == x) out.task[out.ntask++] = task_pack(!lin, !mrows, mrows, true, rank, netL, d);
      }
      ++rank;
    }
  }
}

cudaError_t launch_period(const LaunchShape &sh, const DevProblem *probs, const long long *unit_start,
                          int nprob, long long total, unsigned long long *counter,
                          const Scratch &sc, cudaStream_t st, bool valid = false);
// valid: the validation build of the period kernel (trace, supplied words;
// CTAs of at most 256 threads)
int period_blocks_per_sm(int threads, size_t dyn_smem, bool valid = false);

static_assert(kMaxNet == CUSNA_MAXNET, "network capacity of the kernels and the ABI");
static_assert(kMaxEff == CUSNA_MAXEFF, "effect capacity of the kernels and the ABI");
int multi_blocks_per_sm(int threads, size_t dyn_smem);
cudaError_t launch_multi(const LaunchShape &sh, const DevProblem *nets, const MultiDev &md, int M,
                         unsigned long long *counter, const Scratch &sc, cudaStream_t st);
// Cross-network statistic of M dense own networks a against the dense source
// predictor wp; ar (M*n*W words, type 37) and wr (n*W words, type 36) are
// scratch for packed rows.
cudaError_t launch_cross_stats(const uint8_t *a, const uint8_t *wp, int n, int M, int t,
                               double parm, uint32_t *ar, uint32_t *wr, double *out,
                               cudaStream_t st);
// Rows of dense uint8 matrices (rows x n) packed into W words per row.
cudaError_t launch_pack_rows(const uint8_t *a, long long rows, int n, int W, uint32_t *out,
                             cudaStream_t st);
// Typed (creation / endowment) statistic of M dense end networks.
cudaError_t launch_typed_stats(const uint8_t *a, int n, int M, int etype, const double *F,
                               const uint8_t *x0, const uint8_t *keep, const uint8_t *force,
                               const uint8_t *keepS, const uint8_t *forceS,
                               const uint8_t *miss_m, const uint8_t *miss_m1, double *out,
                               cudaStream_t st);
// sienaGOF distributions of M dense end networks (kind 0 in-degree, 1
// out-degree, 2 geodesic with K = min(largest level, n - 1)); rows (M*n*W
// words) and added (M*(K+1)) are scratch of the geodesic kind.
size_t gof_scratch_words(int n, int M, int kind, int K);
cudaError_t launch_gof(const uint8_t *a, int n, int M, int kind, const int *levls, int nlev,
                       int K, uint32_t *rows, unsigned long long *added, double *out,
                       int smem_optin, cudaStream_t st);

// One theta-premultiplied term table of a plan's problem q, effect e (pool
// offsets of the table and, for lookup tables, of its values).
struct PlanTable {
  int q, e, kind, offt, offd, size;
};
// Before each launch of a plan: advance the epoch (Philox keys) and rebuild the
// term tables from the current parameters.
cudaError_t launch_plan_prologue(DevProblem *probs, const unsigned long long *base_seed, int count,
                                 unsigned long long *epoch, const PlanTable *tabs, int n_tabs,
                                 cudaStream_t st);
// Start values of the count matrices of a launch's problems (their c0).
cudaError_t launch_counts_init(const DevProblem *probs, int nprob, int nmax, bool multi,
                               cudaStream_t st);
long long kernel_launches();  // kernels launched so far by the calling thread
void note_launch();           // counts a launch made outside the wrappers here
// Raises a kernel's dynamic shared memory limit on the current device to at
// least `bytes`; never lowers it (see saom_sim.cu).
cudaError_t raise_dyn_smem(const void *func, size_t bytes);
void set_last_error(const char *msg);  // text of cusna_last_error() for this thread

// A named range on the calling thread's timeline for profilers (NVTX, header
// only: without an attached tool each push and pop is a call that returns).
struct NvtxRange {
  explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange &) = delete;
  NvtxRange &operator=(const NvtxRange &) = delete;
};
cudaError_t launch_netstats(const uint8_t *a, int M, const StatDesc &D, double *out, int sms,
                            cudaStream_t st);
cudaError_t launch_behstats(const int *z, int n, int M, int kb, const int *bty, const uint8_t *xnet,
                            const int *bkdist, double zbar, double brange, double bsimmean,
                            double *out, int sms, cudaStream_t st);
cudaError_t launch_prep_bits(const uint32_t *src, int n, int W, uint32_t *dst, uint32_t *dstc,
                             int def_mode, cudaStream_t st);
cudaError_t launch_prep_desc(const double *d64, const float *d32, size_t cnt, double *dst,
                             cudaStream_t st);
cudaError_t launch_fill_int(int *dst, size_t cnt, int mode, int value, cudaStream_t st);

}  // namespace cusna
