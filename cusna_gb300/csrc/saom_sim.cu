// saom_sim.cu -- kernels of the GB300 SAOM period simulator: the persistent
// period kernel, the standalone statistic kernels and the input-preparation
// kernels. Host code (validation, memory, the C ABI) is in saom_api.cu.
#include "saom_period.cuh"
#include "saom_launch.h"

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

namespace cusna {

// ---- standalone statistics (cusna_network_stats_gpu / behavior_stats_gpu) ----

// A team of four warps (a CTA) per network: pack the dense network into
// word-major rows/cols in shared memory (rows by ballots over coalesced bytes,
// columns by ballots over 32 x 32 bits of the rows), then the same statistic code
// as the period kernel. With one warp per network, whose lane 0 formed and added
// every order-dependent term, 1000 networks of 100 actors and 11 statistics took
// 2.5 ms of the kernel; so 0.59.
constexpr int kNetWarps = 4;
__global__ void __launch_bounds__(32 * kNetWarps) netstats_kernel(
    const uint8_t *__restrict__ a_batch, int M, StatDesc D, double *out, int rows) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int n = D.n, W = D.W;
  Team T;
  T.G = kNetWarps; T.L = 32 * kNetWarps; T.tl = threadIdx.x; T.warp = T.tl >> 5; T.lane = T.tl & 31;
  T.bar = 1;
  uint32_t *R = (uint32_t *)smem;
  uint32_t *Cc = R + (size_t)W * n;
  int *od = (int *)(Cc + (size_t)W * n);
  int *id = od + n;
  double *red = (double *)(((uintptr_t)(id + n) + 15) & ~(uintptr_t)15);
  for (int c = blockIdx.x; c < M; c += gridDim.x) {
    const uint8_t *a = a_batch + (size_t)c * n * n;
    for (int r = T.warp; r < n; r += kNetWarps)
      for (int w = 0; w < W; ++w) {
        const int q = 32 * w + T.lane;
        const uint32_t m = __ballot_sync(kFull, q < n && a[(size_t)r * n + q] != 0);
        if (T.lane == 0) R[w * n + r] = m;
      }
    T.sync();
    for (int w = T.warp; w < W; w += kNetWarps)       // columns' word w: rows 32w..
      for (int cw = 0; cw < W; ++cw) {                // of columns 32cw..
        const int r = 32 * w + T.lane;
        const uint32_t v = r < n ? R[cw * n + r] : 0u;
        uint32_t mine = 0;
#pragma unroll
        for (int b = 0; b < 32; ++b) {
          const uint32_t m = __ballot_sync(kFull, (v >> b) & 1u);
          if (T.lane == b) mine = m;
        }
        if (32 * cw + T.lane < n) Cc[w * n + 32 * cw + T.lane] = mine;
      }
    T.sync();
    for (int x = T.tl; x < n; x += T.L) {
      int o = 0, i2 = 0;
      for (int w = 0; w < W; ++w) { o += __popc(R[w * n + x]); i2 += __popc(Cc[w * n + x]); }
      od[x] = o;
      id[x] = i2;
    }
    T.sync();
    network_stats_team(T, D, R, Cc, od, id, red, rows, out + (size_t)c * D.k);
    T.sync();
  }
}

// Behaviour statistics (src/libcusna_saom_cpu.cpp:768-817): one warp per chain.
// Per-actor terms are formed in parallel; lane 0 adds them in actor order, and
// the avAlt/avSim inner sums run over alters in ascending order, as the
// reference adds them.
__global__ void behstats_kernel(const int *__restrict__ z_batch, int n, int M, int kb,
                                const int *__restrict__ bty, const uint8_t *__restrict__ xnet,
                                const int *__restrict__ bkdist, double zbar, double brange,
                                double bsimmean, double *out) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, tw = threadIdx.x >> 5;
  double *u = (double *)smem + (size_t)tw * 2 * n;
  double *term = u + n;
  for (int c = blockIdx.x * (blockDim.x >> 5) + tw; c < M; c += gridDim.x * (blockDim.x >> 5)) {
    const int *z = z_batch + (size_t)c * n;
    for (int i = lane; i < n; i += 32) {
      const bool ok = bkdist ? bkdist[i] != 0 : true;
      u[i] = ok ? __dsub_rn((double)z[i], zbar) : 0.0;
    }
    __syncwarp();
    for (int e = 0; e < kb; ++e) {
      const int t = bty[e];
      if (t == 2 || t == 3 || t == 4) {
        for (int i = lane; i < n; i += 32) {
          const uint8_t *xr = xnet + (size_t)i * n;
          const bool oki = bkdist ? bkdist[i] != 0 : true;
          double s = 0.0, od = 0.0, nb = 0.0;
          if (t == 2) {
            for (int j = 0; j < n; ++j) if (xr[j]) { od += 1.0; s = __dadd_rn(s, u[j]); }
            term[i] = od <= 0.0 ? 0.0 : __dmul_rn(u[i], __ddiv_rn(s, od));
            if (od <= 0.0) term[i] = -0.0;  // marker: skipped actor
          } else {
            for (int j = 0; j < n; ++j) {
              if (!xr[j]) continue;
              const bool okj = bkdist ? bkdist[j] != 0 : true;
              if (okj) {
                nb += 1.0;
                s = __dadd_rn(s, __dsub_rn(1.0, __ddiv_rn(fabs(__dsub_rn(u[i], u[j])), brange)));
              }
            }
            s = __dsub_rn(s, __dmul_rn(nb, bsimmean));
            if (t == 3) s = nb > 0.0 ? __ddiv_rn(s, nb) : 0.0;
            term[i] = oki ? s : -0.0;
          }
        }
      }
      __syncwarp();
      if (lane == 0) {
        double acc = 0.0;
        if (t == 0) for (int i = 0; i < n; ++i) acc = __dadd_rn(acc, u[i]);
        else if (t == 1) for (int i = 0; i < n; ++i) acc = __dadd_rn(acc, __dmul_rn(u[i], u[i]));
        else if (t >= 2 && t <= 4)
          for (int i = 0; i < n; ++i) {
            // skipped actors contribute nothing (the reference `continue`s);
            // adding -0.0 leaves every partial sum unchanged
            acc = __dadd_rn(acc, term[i]);
          }
        out[(size_t)c * kb + e] = acc;
      }
      __syncwarp();
    }
  }
}

// ---- input preparation ------------------------------------------------------

// Row-major n*W bit rows -> word-major W*n; optionally also the transposed
// matrix (in-rows) word-major. def_offdiag: when src is null, fill with the
// all-ones off-diagonal matrix (the reference's default masks).
__global__ void prep_bits_kernel(const uint32_t *src, int n, int W, uint32_t *dst,
                                 uint32_t *dstc, int def_mode) {
  const size_t total = (size_t)W * n;
  for (size_t x = (size_t)blockIdx.x * blockDim.x + threadIdx.x; x < total;
       x += (size_t)gridDim.x * blockDim.x) {
    const int w = (int)(x / n), r = (int)(x % n);
    uint32_t v = 0, vc = 0;
    for (int b = 0; b < 32; ++b) {
      const int q = 32 * w + b;
      if (q >= n) break;
      int bit_rq, bit_qr;
      if (src) {
        bit_rq = (src[(size_t)r * W + w] >> b) & 1;                 // a[r][q]
        bit_qr = (src[(size_t)q * W + (r >> 5)] >> (r & 31)) & 1;  // a[q][r]
      } else {
        bit_rq = bit_qr = def_mode == 1 ? (q != r) : 0;
      }
      v |= (uint32_t)bit_rq << b;
      vc |= (uint32_t)bit_qr << b;
    }
    if (dst) dst[x] = v;
    if (dstc) dstc[x] = vc;
  }
}

// Start values of the counters that chains hold as matrices, for every problem
// of a launch (block y = problem): cell (i, j) by popcounts, as count_of forms it
// for a ministep of i. Networks w of a multi-network problem are the launch's
// problems w.
__global__ void __launch_bounds__(256) counts_init_kernel(const DevProblem *__restrict__ probs,
                                                          bool multi) {
  const DevProblem &P = probs[blockIdx.y];
  const int n = P.n, W = P.W;
  uint16_t *C = const_cast<uint16_t *>(P.c0);
  for (int c = 0; c < P.cnt.n; ++c) {
    if (!((P.cnt.mask >> c) & 1u)) continue;
    const int list = P.cnt.list[c];
    const uint32_t *A = list == CL_IN ? P.simc
                        : (multi && list >= CL_NET) ? probs[list - CL_NET].simr : P.simr;
    auto rel = [&](int m) -> const uint32_t * {
      return m == CM_ROWS ? P.simc : ((multi && m >= CM_NCOLS) ? probs[m - CM_NCOLS].simr : P.simr);
    };
    const uint32_t *M1 = rel(P.cnt.m1[c]);
    const uint32_t *M2 = P.cnt.m2[c] == CM_NONE ? nullptr : rel(P.cnt.m2[c]);
    for (size_t x = (size_t)blockIdx.x * blockDim.x + threadIdx.x; x < (size_t)n * n;
         x += (size_t)gridDim.x * blockDim.x) {
      const int i = (int)(x / n), j = (int)(x % n);
      int v = 0;
      for (int w = 0; w < W; ++w) {
        const uint32_t a = A[w * n + i];
        v += __popc(a & M1[w * n + j]);
        if (M2) v += __popc(a & M2[w * n + j]);
      }
      C[x] = (uint16_t)v;
    }
    C += cm_size(n);
  }
}

cudaError_t launch_counts_init(const DevProblem *probs, int nprob, int nmax, bool multi,
                               cudaStream_t st) {
  const int bx = (int)std::min<size_t>(((size_t)nmax * nmax + 255) / 256, 1024);
  for (int q = 0; q < nprob; q += 65535) {
    const dim3 grid(bx, std::min(nprob - q, 65535));
    counts_init_kernel<<<grid, 256, 0, st>>>(probs + q, multi);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    note_launch();
  }
  return cudaSuccess;
}

// float64 descriptor with the reference's precedence: the *64 array if given,
// else the float array promoted, else zeros (src/libcusna_saom_cpu.cpp:337-350).
__global__ void prep_desc_kernel(const double *d64, const float *d32, size_t cnt, double *dst) {
  for (size_t x = (size_t)blockIdx.x * blockDim.x + threadIdx.x; x < cnt;
       x += (size_t)gridDim.x * blockDim.x)
    dst[x] = d64 ? d64[x] : (d32 ? (double)d32[x] : 0.0);
}

__global__ void fill_int_kernel(int *dst, size_t cnt, int mode, int value) {
  for (size_t x = (size_t)blockIdx.x * blockDim.x + threadIdx.x; x < cnt;
       x += (size_t)gridDim.x * blockDim.x)
    dst[x] = mode == 0 ? value : (int)x;  // mode 1: identity (act)
}

// ---- launch wrappers used by the host code ----------------------------------

// Kernels launched by this thread (reported through cusna_gpu_options).
thread_local long long g_launches = 0;
long long kernel_launches() { return g_launches; }
void note_launch() { ++g_launches; }
static cudaError_t counted(cudaError_t e) {
  if (e == cudaSuccess) ++g_launches;
  return e;
}

// A kernel's dynamic shared memory limit is one value per function and
// device, shared by every host thread. Setting it to each launch's own size
// would let one thread lower it between another thread's setting and launch,
// and fail that launch; so the limit only rises.
cudaError_t raise_dyn_smem(const void *func, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void *>, size_t> limit;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  size_t &cur = limit[{dev, func}];
  if (bytes <= cur) return cudaSuccess;
  e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) cur = bytes;
  return e;
}

template <int MAXT, bool VALID>
static int blocks_per_sm_t(int threads, size_t dyn_smem) {
  if (raise_dyn_smem((const void *)period_kernel<MAXT, VALID>, dyn_smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, period_kernel<MAXT, VALID>, threads,
                                                    dyn_smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return b;
}

// The validation build exists for CTAs of up to 256 threads only.
int period_blocks_per_sm(int threads, size_t dyn_smem, bool valid) {
  if (valid) return threads <= 256 ? blocks_per_sm_t<256, true>(threads, dyn_smem) : 0;
  return threads <= 256 ? blocks_per_sm_t<256, false>(threads, dyn_smem)
                        : blocks_per_sm_t<512, false>(threads, dyn_smem);
}

cudaError_t launch_period(const LaunchShape &sh, const DevProblem *probs, const long long *unit_start,
                          int nprob, long long total, unsigned long long *counter,
                          const Scratch &sc, cudaStream_t st, bool valid) {
  const int threads = 32 * sh.G * sh.teams_per_cta;
  const size_t dyn = sh.lay.bytes * sh.teams_per_cta;
  if (valid && threads > 256) return cudaErrorInvalidConfiguration;
  auto kern = valid ? period_kernel<256, true>
                    : (threads <= 256 ? period_kernel<256, false> : period_kernel<512, false>);
  cudaError_t e = raise_dyn_smem((const void *)kern, dyn);
  if (e != cudaSuccess) return e;
  kern<<<sh.ctas, threads, dyn, st>>>(probs, unit_start, nprob, total, counter, sh.lay, sh.G,
                                      sc.cols, sc.rows, sc.cols_words, sc.counts, sc.counts_stride);
  return counted(cudaGetLastError());
}

// ---- replayable plans --------------------------------------------------------
// Each launch of a plan simulates with Philox key = the problem's seed plus the
// plan's epoch (64-bit, so epoch 0 is the plain call), then advances the epoch.
__global__ void plan_epoch_kernel(DevProblem *probs, const unsigned long long *base_seed,
                                  int count, unsigned long long *epoch) {
  __shared__ unsigned long long e;
  if (threadIdx.x == 0) e = *epoch;
  __syncthreads();
  for (int q = threadIdx.x; q < count; q += blockDim.x) {
    const unsigned long long s = base_seed[q] + e;
    probs[q].k0 = (uint32_t)(s & 0xFFFFFFFFull);
    probs[q].k1 = (uint32_t)(s >> 32);
  }
  __syncthreads();
  if (threadIdx.x == 0) *epoch = e + 1;
}

// Rebuilds the theta-premultiplied term tables of a plan's problems from the
// current parameter row (one block per table): entry x of effect e's table is
// theta_e * x for a count table and theta_e * value_x for a lookup table,
// rounded as the host builds them.
__global__ void plan_retheta_kernel(const DevProblem *probs, const PlanTable *tabs) {
  const PlanTable T = tabs[blockIdx.x];
  const DevProblem &P = probs[T.q];
  const double th = (double)P.theta[T.e];
  double *tab = const_cast<double *>(P.tab);
  for (int x = blockIdx.y * blockDim.x + threadIdx.x; x < T.size; x += gridDim.y * blockDim.x) {
    const double v = T.kind == K_CNT ? (double)x : tab[T.offd + x];
    tab[T.offt + x] = __dmul_rn(th, v);
  }
}

cudaError_t launch_plan_prologue(DevProblem *probs, const unsigned long long *base_seed, int count,
                                 unsigned long long *epoch, const PlanTable *tabs, int n_tabs,
                                 cudaStream_t st) {
  plan_epoch_kernel<<<1, 256, 0, st>>>(probs, base_seed, count, epoch);
  cudaError_t e = counted(cudaGetLastError());
  if (e != cudaSuccess || n_tabs == 0) return e;
  // eight CTAs a table: a dyadic table has n^2 entries, and one CTA of 128 threads
  // spent the latency of 700 dependent rounds on it at n = 300: 131 us of a 15.2 ms round
  plan_retheta_kernel<<<dim3(n_tabs, 8), 256, 0, st>>>(probs, tabs);
  return counted(cudaGetLastError());
}

cudaError_t launch_netstats(const uint8_t *a, int M, const StatDesc &D, double *out, int sms,
                            cudaStream_t st) {
  const size_t nets = al16((size_t)2 * D.W * D.n * 4 + (size_t)2 * D.n * 4) + 16;
  if (nets + 304 > 200 * 1024) return cudaErrorInvalidValue;
  // scratch for as many statistics at a time as fit (at least two: with them a network
  // that just passes takes 288 bytes more than 200 KiB, which an SM has)
  int rows = D.k < 32 ? D.k : 32;
  while (rows > 2 && nets + stat_scratch(rows) * 8 > 200 * 1024) --rows;
  if (rows < 2) rows = 2;
  const size_t bytes = nets + stat_scratch(rows) * 8;
  cudaError_t e = raise_dyn_smem((const void *)netstats_kernel, bytes);
  if (e != cudaSuccess) return e;
  const int blocks = M < 16 * sms ? M : 16 * sms;
  netstats_kernel<<<blocks, 32 * kNetWarps, bytes, st>>>(a, M, D, out, rows);
  return counted(cudaGetLastError());
}

cudaError_t launch_behstats(const int *z, int n, int M, int kb, const int *bty, const uint8_t *xnet,
                            const int *bkdist, double zbar, double brange, double bsimmean,
                            double *out, int sms, cudaStream_t st) {
  const size_t per = (size_t)2 * n * 8;
  int warps = (int)((200 * 1024) / per);
  if (warps > 8) warps = 8;
  if (warps < 1) return cudaErrorInvalidValue;
  cudaError_t e = raise_dyn_smem((const void *)behstats_kernel, per * warps);
  if (e != cudaSuccess) return e;
  int blocks = (M + warps - 1) / warps;
  if (blocks > 4 * sms) blocks = 4 * sms;
  behstats_kernel<<<blocks, 32 * warps, per * warps, st>>>(z, n, M, kb, bty, xnet, bkdist, zbar,
                                                           brange, bsimmean, out);
  return counted(cudaGetLastError());
}

cudaError_t launch_prep_bits(const uint32_t *src, int n, int W, uint32_t *dst, uint32_t *dstc,
                             int def_mode, cudaStream_t st) {
  const size_t total = (size_t)W * n;
  int blocks = (int)((total + 255) / 256);
  if (blocks > 1024) blocks = 1024;
  if (blocks < 1) blocks = 1;
  prep_bits_kernel<<<blocks, 256, 0, st>>>(src, n, W, dst, dstc, def_mode);
  return counted(cudaGetLastError());
}

cudaError_t launch_prep_desc(const double *d64, const float *d32, size_t cnt, double *dst,
                             cudaStream_t st) {
  if (cnt == 0) return cudaSuccess;
  int blocks = (int)((cnt + 255) / 256);
  if (blocks > 1024) blocks = 1024;
  prep_desc_kernel<<<blocks, 256, 0, st>>>(d64, d32, cnt, dst);
  return counted(cudaGetLastError());
}

cudaError_t launch_fill_int(int *dst, size_t cnt, int mode, int value, cudaStream_t st) {
  if (cnt == 0) return cudaSuccess;
  int blocks = (int)((cnt + 255) / 256);
  if (blocks > 1024) blocks = 1024;
  fill_int_kernel<<<blocks, 256, 0, st>>>(dst, cnt, mode, value);
  return counted(cudaGetLastError());
}

}  // namespace cusna
