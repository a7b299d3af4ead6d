// Learned warm start of the MHD inversion (u2p) on independent cells.
//
// KORAL's u2p (u2p.c:176-485) starts its Newton iteration on
// W = w gamma^2 from the primitives it is handed (u2p.c:2093-2112), and
// tries the energy equation first and the entropy equation when that
// fails.  Here the same network as the implicit solve's warm start
// (16 -> 128 -> 128 -> 8, BF16 tensor-core kernels in kgpu_mlp.cu) predicts
// from the conserved state, the guess and the metric (u2p_features in
// kgpu_mlp.cuh):
//   output 0  ln(W / W_guess), W the root the plain inversion converges to
//   output 1  a score (trained on 0/1) that the energy equation fails
// and the inversion starts from W_guess exp(output 0): with the energy
// equation unless the score says it fails, then the entropy equation; if
// neither converges from the prediction, the reference's inversion runs
// from the reference's guess (the fallback), so the set of cells that
// invert is never smaller than the reference's.  Every Newton step is the
// unchanged FP64 one and ends on the same residual test (U2PCONV).
//
// Without a prediction it is the reference's u2p itself (the bits of
// kgpu_u2p_cells), with its Newton iterations counted, in two launches.
#include <cuda_runtime.h>
#include <string.h>

#include "../../include/koral_b200.h"
#include "kgpu_mlp.cuh"
#include "kgpu_slots.h"

using namespace kgpu;

int kgpu_report_cuda(const char *what, cudaError_t e);

namespace {

#define WCK(call)                                              \
  do {                                                         \
    cudaError_t e_ = (call);                                   \
    if (e_ != cudaSuccess) return kgpu_report_cuda(#call, e_); \
  } while (0)

struct U2PParams {
  double gamma, u2pconv, rhofloor;
};

__device__ inline void cell_geom(const double *g20, const double *G20, long i, Geom &g) {
  RadGeom rg;
  rad_geom(g20 + 20 * i, G20 + 20 * i, rg);
  g = rg.g;
}

__device__ inline Grid u2p_grid(const U2PParams &P) {
  Grid G;
  memset(&G, 0, sizeof(G));
  G.gamma = P.gamma;
  G.u2pconv = P.u2pconv;
  G.rhofloor = P.rhofloor;
  G.nv = NVMAX;
  return G;
}

// u2p_solver_W from a given initial W (the bracketing, Newton steps and
// final checks of u2p.c:2117-2292); counts Newton steps and W evaluations
__device__ int solve_from(const Grid &G, const double *uu, double *pp, const Geom &g, int Etype, double W,
                          unsigned &iters, unsigned &fevals) {
  U2PState s;
  u2p_setup(uu, g, s);
  int iter = 0;
  const int r = u2p_solve_w(G.gamma, G.u2pconv, Etype, s.c, W, iter, 1 << 30, 1 << 30, &fevals, 0u);
  iters += (unsigned)iter;
  if (r < 0) return r;
  return u2p_final(G.gamma, s, W, iter, uu, pp, g);
}

// u2p (u2p.c:176-485) with both solves started from W0 when W0 > 0, from
// the reference's guess (the primitives pp) otherwise; the same sequence
// of operations as kgpu::u2p when W0 <= 0
__device__ int u2p_counted(const Grid &G, const double *uu0, double *pp, const Geom &g, int &fixup, double W0,
                           bool skip_energy, unsigned &iters, unsigned &fevals) {
  double uu[NVMAX], ppbak[NVMAX];
  for (int iv = 0; iv < NVMAX; iv++) {
    uu[iv] = uu0[iv];
    ppbak[iv] = pp[iv];
  }
  int ret = 0, u2pret = -1;
  if (uu[0] / g.gdet < 0.) {
    pp[0] = G.rhofloor;
    uu[0] = G.rhofloor * g.gdet;
    ret = -2;
  }
  if (!skip_energy) u2pret = solve_from(G, uu, pp, g, 0, W0 > 0. ? W0 : u2p_initial_w(G.gamma, pp, g), iters, fevals);
  if (u2pret < 0) {
    ret = -1;
    // the reference's entropy solve reads its guess from pp again (which a
    // failed energy solve may have changed: u2p.c:2281-2293 writes the
    // primitives before the negative-density check)
    u2pret = solve_from(G, uu, pp, g, 1, W0 > 0. ? W0 : u2p_initial_w(G.gamma, pp, g), iters, fevals);
    if (u2pret < 0) ret = -2;
  }
  if (u2pret < 0) {
    ret = -3;
    for (int iv = 0; iv < NVMAX; iv++) pp[iv] = ppbak[iv];
  }
  fixup = (ret < -1) ? 1 : 0;
  return ret;
}

// ---------------------------------------------------------------------------
// The inversion without a prediction, in two launches.  One thread per cell
// through both equations made every warp as slow as its slowest cell: on
// 1048576 magnetised cells, 1% of which end in the entropy equation, 4.9 of
// 32 lanes were active on average and a launch took 3.8 ms.  Now k_u2p_first
// gives every cell the energy equation with the limits of the grid's first
// pass and marks the cells that need more in their status; k_u2p_rest gathers
// those, block by block over a range of cells, and gives the paused solves a
// warp each and the entropy solves a thread each, with the same limits, and
// then a warp each.  Per cell the same steps are taken, so results and
// counters are the same.  No memory besides the outputs is needed.
// ---------------------------------------------------------------------------
enum : int { CELL_PAUSED = 1001, CELL_ENTROPY = 1002, CELL_WHOLE = 1003 };   // no status u2p returns
constexpr int FIRST_STEPS = 8, FIRST_HALVINGS = 4;

__device__ inline void add_stats(unsigned long long *stats, unsigned it, unsigned fell, unsigned fe) {
  const unsigned m = __activemask();
  const unsigned a = __reduce_add_sync(m, it), b = __reduce_add_sync(m, fell), c = __reduce_add_sync(m, fe);
  if ((threadIdx.x & 31) == __ffs(m) - 1) {
    if (a) atomicAdd(&stats[0], (unsigned long long)a);
    if (b) atomicAdd(&stats[1], (unsigned long long)b);
    if (c) atomicAdd(&stats[2], (unsigned long long)c);
  }
}

// the cell as u2p starts on it; true where its density was negative
__device__ inline bool cell_load(const Grid &G, int nv, const double *uu, const double *pp, long i, const Geom &g,
                                 double *u, double *p) {
  for (int iv = 0; iv < NVMAX; iv++) {
    u[iv] = uu[i * nv + iv];
    p[iv] = pp[i * nv + iv];
  }
  if (!(u[0] / g.gdet < 0.)) return false;
  p[0] = G.rhofloor;
  u[0] = G.rhofloor * g.gdet;
  return true;
}
__device__ inline void cell_store(int nv, double *pp, long i, const double *p, int ret, int it, int *status,
                                  int *fixup, int *iters) {
  if (ret != -3)
    for (int iv = 0; iv < NVMAX; iv++) pp[i * nv + iv] = p[iv];   // a failure keeps the guess
  status[i] = ret;
  fixup[i] = ret < -1 ? 1 : 0;
  if (iters) iters[i] = it;
}

__global__ void __launch_bounds__(128, 4) k_u2p_first(U2PParams P, int n, int nv, const double *uu, double *pp,
                                                      const double *g20, const double *G20, int *status, int *fixup,
                                                      int *iters, unsigned long long *stats) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Grid G = u2p_grid(P);
  Geom g;
  cell_geom(g20, G20, i, g);
  double u[NVMAX], p[NVMAX];
  const bool negrho = cell_load(G, nv, uu, pp, i, g, u, p);
  U2PState s;
  u2p_setup(u, g, s);
  double W = u2p_initial_w(G.gamma, p, g);
  int it = 0;
  unsigned fe = 0;
  int r = u2p_solve_w(G.gamma, G.u2pconv, 0, s.c, W, it, FIRST_STEPS, FIRST_HALVINGS, &fe);
  const bool paused = r == U2P_PAUSED;
  if (r == 0) r = u2p_final(G.gamma, s, W, it, u, p, g);
  if (paused) {
    status[i] = CELL_PAUSED;   // its solve is done again from the start
  } else if (r < 0) {
    // what a failed solve leaves in the primitives is read by the next: only
    // the check on the density fails after they are set
    status[i] = r == -105 ? CELL_WHOLE : CELL_ENTROPY;
    fixup[i] = it;
  } else {
    cell_store(nv, pp, i, p, negrho ? -2 : 0, it, status, fixup, iters);
  }
  const bool count = !paused && r != -105;
  if (stats) add_stats(stats, count ? it : 0, 0, count ? fe : 0);
}

// a warp on the whole solve of equation Etype of one cell; every lane returns
// the same values
__device__ inline int solve_warp(const Grid &G, const double *u, double *p, const Geom &g, int Etype, int &it,
                                 unsigned &fe) {
  U2PState s;
  u2p_setup(u, g, s);
  double W = u2p_initial_w(G.gamma, p, g);
  U2PF F;
  if (u2p_bracket(G.gamma, Etype, s.c, W, F, &fe)) return -150;
  int k = 0;
  const int r = u2p_newton_warp(G.gamma, G.u2pconv, Etype, s.c, W, k, F, true, &fe);
  it += k;
  if (r < 0) return r;
  return u2p_final(G.gamma, s, W, k, u, p, g);
}

// cells a block of the second launch looks over: 1.47 ms for 2^20 cells at
// 1024, 1.55 at 512 (fewer hard cells to a warp), 1.60 at 2048 (fewer blocks)
constexpr int REST_THREADS = 128, REST_RANGE = 1024;

__global__ void __launch_bounds__(REST_THREADS) k_u2p_rest(U2PParams P, int n, int nv, int range, const double *uu,
                                                           double *pp, const double *g20, const double *G20,
                                                           int *status, int *fixup, int *iters,
                                                           unsigned long long *stats) {
  __shared__ int cell[REST_RANGE];   // paused from the front, to the entropy equation from the back
  __shared__ int na, nb;
  const Grid G = u2p_grid(P);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i0 = blockIdx.x * range, i1 = i0 + range < n ? i0 + range : n;
  if (tid == 0) na = nb = 0;
  __syncthreads();
  for (int i = i0 + tid; i < i1; i += REST_THREADS) {
    const int st = status[i];
    if (st == CELL_PAUSED) cell[atomicAdd(&na, 1)] = i;
    else if (st == CELL_ENTROPY || st == CELL_WHOLE) cell[range - 1 - atomicAdd(&nb, 1)] = i;
  }
  __syncthreads();
  // paused energy solves, a warp each; one that fails is marked for the
  // entropy equation
  const int n1 = na, n2 = nb;
  for (int q = warp; q < n1; q += REST_THREADS / 32) {
    const int i = cell[q];
    Geom g;
    cell_geom(g20, G20, i, g);
    double u[NVMAX], p[NVMAX];
    const bool negrho = cell_load(G, nv, uu, pp, i, g, u, p);
    int it = 0;
    unsigned fe = 0;
    const int r = solve_warp(G, u, p, g, 0, it, fe);
    __syncwarp();
    if (lane == 0) {
      if (r < 0) {
        status[i] = r == -105 ? CELL_WHOLE : CELL_ENTROPY;
        fixup[i] = it;
      } else {
        cell_store(nv, pp, i, p, negrho ? -2 : 0, it, status, fixup, iters);
      }
      if (stats && !(r == -105)) add_stats(stats, it, 0, fe);
    }
    __syncwarp();
  }
  __syncthreads();
  // entropy solves, a thread each, over both lists; the paused ones are
  // marked and stay for the warps
  const int total = n1 + n2;
  for (int q = tid; q < total; q += REST_THREADS) {
    const int i = cell[q < n2 ? range - 1 - q : q - n2];
    const int st = status[i];
    if (st == CELL_WHOLE || st == CELL_ENTROPY) {
      Geom g;
      cell_geom(g20, G20, i, g);
      double u[NVMAX], p[NVMAX];
      if (st == CELL_WHOLE) {
        for (int iv = 0; iv < NVMAX; iv++) {
          u[iv] = uu[(long)i * nv + iv];
          p[iv] = pp[(long)i * nv + iv];
        }
        int fix = 0;
        unsigned it = 0, fe = 0;
        const int ret = u2p_counted(G, u, p, g, fix, -1., false, it, fe);
        cell_store(nv, pp, i, p, ret, (int)it, status, fixup, iters);
        if (stats) add_stats(stats, it, 0, fe);
      } else {
        cell_load(G, nv, uu, pp, i, g, u, p);
        U2PState s;
        u2p_setup(u, g, s);
        double W = u2p_initial_w(G.gamma, p, g);
        int it = 0;
        unsigned fe = 0;
        int r = u2p_solve_w(G.gamma, G.u2pconv, 1, s.c, W, it, FIRST_STEPS, FIRST_HALVINGS, &fe);
        const bool paused = r == U2P_PAUSED;
        if (r == 0) r = u2p_final(G.gamma, s, W, it, u, p, g);
        if (paused) {
          status[i] = CELL_PAUSED;
        } else {
          cell_store(nv, pp, i, p, r < 0 ? -3 : -1, fixup[i] + it, status, fixup, iters);
          if (stats) add_stats(stats, it, 0, fe);
        }
      }
    }
  }
  __syncthreads();
  for (int q = warp; q < total; q += REST_THREADS / 32) {
    const int i = cell[q < n2 ? range - 1 - q : q - n2];
    if (status[i] != CELL_PAUSED) continue;
    Geom g;
    cell_geom(g20, G20, i, g);
    double u[NVMAX], p[NVMAX];
    cell_load(G, nv, uu, pp, i, g, u, p);
    int it = 0;
    unsigned fe = 0;
    const int r = solve_warp(G, u, p, g, 1, it, fe);
    __syncwarp();   // every lane has read the status
    if (lane == 0) {
      cell_store(nv, pp, i, p, r < 0 ? -3 : -1, fixup[i] + it, status, fixup, iters);
      if (stats) add_stats(stats, it, 0, fe);
    }
    __syncwarp();
  }
}

// The inversion from a prediction, one thread per cell
__global__ void k_u2p_warm_cells(U2PParams P, int n, int nv, const double *uu, double *pp, const double *g20,
                                 const double *G20, const float *ypred, float wgate, float sgate, int *status,
                                 int *fixup, int *iters, unsigned long long *stats) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned it = 0, fe = 0, fell = 0;
  if (i < n) {
    const Grid G = u2p_grid(P);
    Geom g;
    cell_geom(g20, G20, i, g);
    double u[NVMAX], p[NVMAX], p0[NVMAX];
    for (int iv = 0; iv < NVMAX; iv++) {
      u[iv] = uu[(long)i * nv + iv];
      p[iv] = p0[iv] = pp[(long)i * nv + iv];
    }
    int fix = 0;
    const float *y = ypred + (long)i * MLP_OUTP;
    // a predicted change of W smaller than wgate is within the network's
    // own error: the guess's W is kept; the energy equation is skipped
    // where the score passes sgate
    const double W0 = fabsf(y[0]) >= wgate ? u2p_warm_w(G.gamma, p0, g, y[0]) : u2p_initial_w(G.gamma, p0, g);
    int ret = W0 > 0. ? u2p_counted(G, u, p, g, fix, W0, y[1] > sgate, it, fe) : -3;
    if (ret < -1) {
      // fallback: the reference's inversion from the reference's guess
      fell = 1;
      for (int iv = 0; iv < NVMAX; iv++) p[iv] = p0[iv];
      ret = u2p_counted(G, u, p, g, fix, -1., false, it, fe);
    }
    for (int iv = 0; iv < NVMAX; iv++) pp[(long)i * nv + iv] = p[iv];
    status[i] = ret;
    fixup[i] = fix;
    if (iters) iters[i] = (int)it;
  }
  if (stats) {
    // per-warp sums, one atomic per warp and counter
    unsigned long long a = it, b = fell, c = fe;
    for (int o = 16; o; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
      c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if ((threadIdx.x & 31) == 0) {
      if (a) atomicAdd(&stats[0], a);
      if (b) atomicAdd(&stats[1], b);
      if (c) atomicAdd(&stats[2], c);
    }
  }
}

__global__ void k_u2p_features(U2PParams P, int n, int nv, const double *uu, const double *pp, const double *g20,
                               const double *G20, float *X) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Geom g;
  cell_geom(g20, G20, i, g);
  float x[MLP_IN];
  u2p_features(P.gamma, uu + (long)i * nv, pp + (long)i * nv, g, x);
  for (int f = 0; f < MLP_IN; f++) X[(long)i * MLP_IN + f] = x[f];
}

__global__ void k_u2p_targets(U2PParams P, int n, int nv, const double *pp0, const double *pp1, const double *g20,
                              const double *G20, const int *status, float *T) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Geom g;
  cell_geom(g20, G20, i, g);
  double t[MLP_OUT];
  const bool ok = status[i] == 0 || status[i] == -1;
  u2p_targets(P.gamma, pp0 + (long)i * nv, pp1 + (long)i * nv, g, status[i], t);
  for (int o = 0; o < MLP_OUT; o++) T[(long)i * MLP_OUT + o] = ok ? (float)t[o] : __int_as_float(0x7fc00000);
}

bool params_of(const kgpu_config *cfg, int nv, U2PParams &P) {
  if (!cfg || nv < NVMAX) return false;
  if (!(cfg->gamma > 1.) || !(cfg->u2pconv > 0.)) return false;
  P.gamma = cfg->gamma;
  P.u2pconv = cfg->u2pconv;
  P.rhofloor = cfg->rhofloor;
  return true;
}

// The counters of a call that reports them: a row of an array of the module,
// held from the call's start until its stream has been synchronised.  The
// array belongs to the device's context and its address is asked for in every
// call, so no device pointer outlives what it points to.  With every row held
// by other threads' calls the call allocates its own, as all did at first: a
// stream-ordered allocation goes back to the driver at every synchronisation,
// and mapping it anew costs a few hundred microseconds.
__device__ unsigned long long g_counters[Slots::N][3];
Slots g_counter_rows;

class CallCounters {
 public:
  explicit CallCounters(cudaStream_t s) : s_(s) {}
  ~CallCounters() {
    if (row_ < 0 && !p_) return;
    if (!synced_) cudaStreamSynchronize(s_);   // a call that failed: what it enqueued may still run
    if (row_ >= 0) g_counter_rows.give(row_);
    else cudaFreeAsync(p_, s_);
  }
  // cleared on the stream
  cudaError_t open(unsigned long long **p) {
    cudaError_t e;
    row_ = g_counter_rows.take();
    if (row_ >= 0) {
      void *base = nullptr;
      if ((e = cudaGetSymbolAddress(&base, g_counters)) != cudaSuccess) return e;
      *p = (unsigned long long *)base + 3 * row_;
    } else {
      if ((e = cudaMallocAsync(&p_, 3 * sizeof(unsigned long long), s_)) != cudaSuccess) return e;
      *p = (unsigned long long *)p_;
    }
    return cudaMemsetAsync(*p, 0, 3 * sizeof(unsigned long long), s_);
  }
  void synced() { synced_ = true; }

 private:
  cudaStream_t s_;
  int row_ = -1;
  void *p_ = nullptr;
  bool synced_ = false;
};

}  // namespace

extern "C" int kgpu_u2p_features_device(int n, const kgpu_config *cfg, int nv, const double *uu, const double *pp,
                                        const double *g, const double *G, float *X, void *stream) {
  U2PParams P;
  if (n < 0 || !params_of(cfg, nv, P) || (n > 0 && (!uu || !pp || !g || !G || !X))) return KGPU_EINVAL;
  if (n == 0) return 0;
  k_u2p_features<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>(P, n, nv, uu, pp, g, G, X);
  WCK(cudaGetLastError());
  return 0;
}

extern "C" int kgpu_u2p_targets_device(int n, const kgpu_config *cfg, int nv, const double *pp, const double *pp1,
                                       const double *g, const double *G, const int *status, float *T,
                                       void *stream) {
  U2PParams P;
  if (n < 0 || !params_of(cfg, nv, P) || (n > 0 && (!pp || !pp1 || !g || !G || !status || !T))) return KGPU_EINVAL;
  if (n == 0) return 0;
  k_u2p_targets<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>(P, n, nv, pp, pp1, g, G, status, T);
  WCK(cudaGetLastError());
  return 0;
}

extern "C" int kgpu_u2p_cells_device(int n, const kgpu_config *cfg, int nv, const double *uu, double *pp,
                                     const double *g, const double *G, const float *ypred, float wgate, float sgate,
                                     int *status, int *fixup, int *iters, void *stream, unsigned long long *stats,
                                     int nstats) {
  U2PParams P;
  if (n < 0 || !params_of(cfg, nv, P) || nstats < 0 || nstats > 3 || (nstats > 0 && !stats)) return KGPU_EINVAL;
  if (!(wgate >= 0.f) || !(sgate >= 0.f)) return KGPU_EINVAL;
  if (n > 0 && (!uu || !pp || !g || !G || !status || !fixup)) return KGPU_EINVAL;
  for (int k = 0; k < nstats; k++) stats[k] = 0;
  if (n == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  unsigned long long *dstats = nullptr;
  CallCounters counters(s);
  if (nstats > 0) WCK(counters.open(&dstats));
  cudaError_t e;
  if (ypred) {
    k_u2p_warm_cells<<<(n + 127) / 128, 128, 0, s>>>(P, n, nv, uu, pp, g, G, ypred, wgate, sgate, status, fixup, iters,
                                                      dstats);
    e = cudaGetLastError();
  } else {
    k_u2p_first<<<(n + 127) / 128, 128, 0, s>>>(P, n, nv, uu, pp, g, G, status, fixup, iters, dstats);
    e = cudaGetLastError();
    if (e == cudaSuccess) {
      // a range per block: as many blocks as two per SM hold, so that a
      // block's few hard cells fill more of its lanes, down to a range of 128
      int dev = 0, sms = 148;
      if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      int range = (n + 2 * sms - 1) / (2 * sms);
      range = range < REST_THREADS ? REST_THREADS : (range > REST_RANGE ? REST_RANGE : range);
      k_u2p_rest<<<(n + range - 1) / range, REST_THREADS, 0, s>>>(P, n, nv, range, uu, pp, g, G, status, fixup, iters,
                                                                   dstats);
      e = cudaGetLastError();
    }
  }
  if (dstats) {
    unsigned long long h[3] = {0, 0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, dstats, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && (e = cudaStreamSynchronize(s)) == cudaSuccess) counters.synced();
    for (int k = 0; k < nstats; k++) stats[k] = h[k];
  }
  WCK(e);
  return 0;
}
