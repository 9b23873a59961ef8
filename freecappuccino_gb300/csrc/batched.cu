// Batched DPCG: several independent pressure solves of uneven sizes -- each bound to its
// own context (mesh, sliced matrix) -- in one persistent cooperative kernel, captured in
// a CUDA graph.  No reference counterpart as a batch: every system follows dpcg.f90:3-154
// exactly as fcg_dpcg does (same recurrence, constants and L1 stop test per system).
//
// Work is a list of items, runs of 32-row slices, numbered over the systems still
// iterating.  The kernel walks all systems in lockstep phases -- initial residual; then per
// CG iteration p-update | SpMV | update -- separated by a grid-wide barrier.  In every
// phase each CTA takes an equal, consecutive share of the items, so a large system uses the
// whole GPU, small ones share it, and a CTA meets one system or two: it forms one partial
// sum per system it meets.  The CTA that arrives last at the barrier adds every system's
// partials in CTA order and updates the systems' scalars before it opens the barrier, so a
// solve gives the same bits run after run.  A system that meets its stop test drops out and
// the items are numbered anew; the kernel ends when none is left.
//
// What bounds it: memory latency in the phases, hidden by resident warps (the kernel is held
// to 40 registers, six CTAs an SM), and three barriers of 2 to 5 us a sweep.  12 systems of
// 7.9 M cells in all, a sweep: p 47, SpMV 147, update 101 us.  With one partial sum, block barrier
// and ticket per item and two CTAs an SM a sweep took 811 us, and at its best setting
// (five CTAs, items of 128 slices) 360; rows of eight loads issued together, which need 64
// registers, 444.
//
// The grid barrier spins with a bounded number of polls; a CTA that gives up sets the
// error flag, which ends every CTA at its next barrier, and the call returns
// FCG_ERR_TIMEOUT.  The item size (slices per item) and the CTAs per SM are picked by
// fcg_batch_autotune, which times every candidate on the caller's systems.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <set>
#include <string>
#include <vector>

#include "fcg_internal.h"
#include "krylov_common.cuh"
#include "launch.h"

namespace fcg {
namespace {

constexpr int kMaxBatch = 64;
constexpr int kResident = 6;  // CTAs an SM the kernel's registers are held to

// One system of the batch (device-resident; the host writes the inputs before a solve).
struct BSys {
  SellView sv;
  int n, nitems, nsw;
  const double *val, *invd, *su;
  double *x, *res, *p, *q;
  double sor, small, tol;
  double res0, resl, sk, s0, bet, alf, l2r, l2b;
  int iter, active, converged, status, early;
};

struct BCtl {
  unsigned int count, gen;  // grid barrier
  int err;                  // 1: a barrier wait gave up, 2: loop bound exceeded
  int nactive;              // systems still iterating
};

// The items of the systems still iterating, base[k] .. base[k+1] system k's, in equal shares:
// q items for every CTA and one more for the first rem.
struct Split {
  int base[kMaxBatch + 1], n[kMaxBatch];
  int q, rem;
  __device__ __forceinline__ int begin(int b) const { return b * q + min(b, rem); }
  // the CTA whose share holds `item`
  __device__ __forceinline__ int cta_of(int item) const {
    return item < rem * (q + 1) ? item / (q + 1) : rem + (item - rem * (q + 1)) / q;
  }
};

__device__ void make_split(Split &sp, const BSys *sys, int nsys, bool all) {
  __syncthreads();
  for (int k = threadIdx.x; k < nsys; k += blockDim.x)
    sp.n[k] = all || __ldcg(&sys[k].active) ? sys[k].nitems : 0;
  __syncthreads();
  for (int k = threadIdx.x; k <= nsys; k += blockDim.x) {
    int t = 0;
    for (int j = 0; j < k; ++j) t += sp.n[j];
    sp.base[k] = t;
    if (k == nsys) {
      sp.q = t / (int)gridDim.x;
      sp.rem = t % (int)gridDim.x;
    }
  }
  __syncthreads();
}

// Runs f(k, s0, s1) on this CTA's share: slices [s0, s1) of system k.
template <class F>
__device__ __forceinline__ void for_share(const Split &sp, const BSys *sys, int nsys, int spi,
                                          F &&f) {
  int i = sp.begin(blockIdx.x);
  const int end = sp.begin(blockIdx.x + 1);
  for (int k = 0; i < end; ++k) {
    if (sp.base[k + 1] <= i) continue;
    const int e = min(end, sp.base[k + 1]);
    f(k, (i - sp.base[k]) * spi,
      (int)min((long long)(e - sp.base[k]) * spi, (long long)sys[k].sv.nslices));
    i = e;
  }
}

// This CTA's block sums of system k: part[(k gridDim + CTA) 2 ..].
template <int NV>
__device__ __forceinline__ void put_partial(double (&v)[NV], double *part, int k,
                                            double (*sh)[kTPB]) {
  block_sum<NV>(v, sh);
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) part[((long long)k * gridDim.x + blockIdx.x) * 2 + q] = v[q];
}

// Grid-wide barrier with a bounded wait.  The CTA that arrives last runs `last` (all its
// threads) before the others go on: everything they wrote is visible to it.  Returns false
// when any CTA has given up.
template <class F>
__device__ __forceinline__ bool grid_sync(BCtl *ctl, long long limit, F &&last) {
  __shared__ int state_sh;  // 0: gave up, 1: passed, 2: last to arrive
  __shared__ unsigned int gen_sh;
  __syncthreads();
  if (threadIdx.x == 0) {
    state_sh = 0;
    if (!*(volatile int *)&ctl->err) {
      const unsigned int g = *(volatile unsigned int *)&ctl->gen;
      gen_sh = g;
      __threadfence();
      state_sh = atomicAdd(&ctl->count, 1u) == gridDim.x - 1 ? 2 : 1;
    }
  }
  __syncthreads();
  if (state_sh == 2) {
    __threadfence();
    last();
    __syncthreads();
    if (threadIdx.x == 0) {
      ctl->count = 0u;
      __threadfence();
      atomicAdd(&ctl->gen, 1u);
    }
  } else if (state_sh == 1 && threadIdx.x == 0) {
    long long polls = 0;
    while (*(volatile unsigned int *)&ctl->gen == gen_sh) {
      const bool over = ++polls > limit;
      if (over) atomicCAS(&ctl->err, 0, 1);
      if (over || *(volatile int *)&ctl->err) {
        state_sh = 0;
        break;
      }
      __nanosleep(20);
    }
  }
  __syncthreads();
  __threadfence();
  return state_sh != 0;
}
__device__ __forceinline__ bool grid_sync(BCtl *ctl, long long limit) {
  return grid_sync(ctl, limit, [] {});
}

// In the last CTA of a barrier: every system's partials added in CTA order, then fin(k, sums)
// by one lane.  A system has `width` lanes, a warp while eight systems or fewer are there and
// less of one for more, so that all systems are closed at the same time: what a close costs is
// latency (the loads, the FP64 sums' and quotients' chains), and a warp a system took 48
// systems of 12^3 six rounds of it (90 us a sweep).
static_assert(kMaxBatch * 4 <= kTPB, "four lanes a system at least");
template <class F>
__device__ __forceinline__ void sum_systems(const Split &sp, int nsys, const double *part, F &&fin) {
  int width = 32;
  while (width * nsys > kTPB) width >>= 1;
  const int k = threadIdx.x / width, lane = threadIdx.x & (width - 1);
  const bool on = k < nsys && sp.n[k] > 0;
  const int b0 = on ? sp.cta_of(sp.base[k]) : 0, b1 = on ? sp.cta_of(sp.base[k + 1] - 1) : -1;
  const double *pk = part + (long long)k * gridDim.x * 2;
  double v[2] = {0.0, 0.0};
  for (int b = b0 + lane; b <= b1; b += 8 * width) {
    double2 t[8];  // the loads of eight partials in flight together
#pragma unroll
    for (int u = 0; u < 8; ++u)
      t[u] = b + width * u <= b1
                 ? __ldcg(reinterpret_cast<const double2 *>(pk + 2 * (b + width * u)))
                 : make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      v[0] += t[u].x;
      v[1] += t[u].y;
    }
  }
  __syncwarp();
  for (int o = width >> 1; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 2; ++q) v[q] += __shfl_down_sync(0xffffffffu, v[q], o, width);
  if (on && lane == 0) fin(k, v);
}

// Row sum of A x for lane `lane` of slice `slice` (FP64, slot order = CSR column order).
// x is written by other CTAs between phases, so it is read with plain coherent loads.
__device__ __forceinline__ double brow(const SellView &s, int n, const double *__restrict__ val,
                                       const double *x, int slice, int lane) {
  const long long base = __ldg(&s.ptr[slice]) + lane;
  const int w = __ldg(&s.width[slice]), op = __ldg(&s.offp[slice]);
  double acc = 0.0;
  if (__ldg(&s.kind[slice]) == 0) {
    const int row = slice * 32 + lane;
    for (int j = 0; j < w; ++j) {
      int c = row + __ldg(&s.off[op + j]);
      c = c < 0 ? 0 : (c >= n ? n - 1 : c);
      acc += __ldg(&val[base + (long long)j * 32]) * x[c];
    }
  } else {
    for (int j = 0; j < w; ++j)
      acc += __ldg(&val[base + (long long)j * 32]) * x[__ldg(&s.off[op + 32 * j + lane])];
  }
  return acc;
}

__device__ __noinline__ void fin_init(BSys &S, BCtl *ctl, double l1, double sk) {
  S.res0 = l1;
  S.resl = l1;
  S.iter = 0;
  S.s0 = (double)1.e20f;  // dpcg.f90:76
  S.sk = sk;
  S.bet = sk / S.s0;
  S.converged = 0;
  if (!isfinite(l1)) S.status = FCG_ERR_NONFINITE;
  S.active = !(S.nsw <= 0 || (S.early && l1 < S.tol) || S.status);  // dpcg.f90:66-70
  if (!S.active) atomicSub(&ctl->nactive, 1);
}

__device__ __noinline__ void fin_spmv(BSys &S, double pq) {
  S.alf = S.sk / pq;  // dpcg.f90:119-121
  if (!isfinite(S.alf)) {
    S.status = FCG_ERR_NONFINITE;
    S.alf = 0.0;
  }
}

__device__ __noinline__ void fin_update(BSys &S, BCtl *ctl, double resl, double sk_new) {
  const int it = S.iter + 1;
  S.iter = it;
  S.resl = resl;
  S.s0 = S.sk;  // dpcg.f90:132
  S.sk = sk_new;
  S.bet = sk_new / S.s0;
  if (resl / (S.res0 + S.small) < S.sor) S.converged = 1;  // dpcg.f90:139-142
  if (!isfinite(resl)) S.status = FCG_ERR_NONFINITE;
  if (S.converged || it >= S.nsw || S.status) {
    S.active = 0;
    atomicSub(&ctl->nactive, 1);
  }
}

// The phases' row loops and the barriers' sums are functions of their own, so that each is
// allocated registers for itself: inlined into the kernel they spilled.

// res = su - A x of slices [s0, s1), or only its squares (FINAL) with those of su.
template <bool FINAL>
__device__ __noinline__ double2 residual_rows(const BSys &S, int s0, int s1) {
  const int lane = threadIdx.x & 31;
  double2 v = {0.0, 0.0};
  for (int slice = s0 + (threadIdx.x >> 5); slice < s1; slice += kWarps) {
    const int r = slice * 32 + lane;
    const double ax = brow(S.sv, S.n, S.val, S.x, slice, lane);
    if (r < S.n) {
      const double rr = S.su[r] - ax;
      if (FINAL) {
        v.x += rr * rr;
        v.y += S.su[r] * S.su[r];
      } else {
        S.res[r] = rr;
        v.x += fabs(rr);
        v.y += rr * (rr * __ldg(&S.invd[r]));
      }
    }
  }
  return v;
}

// q = A p of slices [s0, s1), returns p.q
__device__ __noinline__ double spmv_rows(const BSys &S, int s0, int s1) {
  const int lane = threadIdx.x & 31;
  const SellView sv = S.sv;
  const int n = S.n;
  const double *val = S.val, *p = S.p;
  double *q = S.q, v = 0.0;
  for (int slice = s0 + (threadIdx.x >> 5); slice < s1; slice += kWarps) {
    const int r = slice * 32 + lane;
    const double t = brow(sv, n, val, p, slice, lane);
    if (r < n) {
      q[r] = t;
      v += p[r] * t;
    }
  }
  return v;
}

enum Phase { kInit, kSpmv, kUpdate, kFinal };

__device__ __noinline__ void close_phase(int phase, BSys *sys, BCtl *ctl, const Split &sp, int nsys,
                                         const double *part) {
  sum_systems(sp, nsys, part, [&](int k, double *v) {
    if (phase == kInit) fin_init(sys[k], ctl, v[0], v[1]);
    if (phase == kSpmv) fin_spmv(sys[k], v[0]);
    if (phase == kUpdate) fin_update(sys[k], ctl, v[0], v[1]);
    if (phase == kFinal) {
      sys[k].l2r = v[0];
      sys[k].l2b = v[1];
    }
  });
}

__global__ void __launch_bounds__(kTPB, kResident)
    k_batch_dpcg(BSys *sys, int nsys, int spi, double *part, BCtl *ctl, int max_loops,
                 long long spin_limit, int absent_block) {
  __shared__ double sh[2][kTPB];
  __shared__ Split sp;
  // diagnostics only (fcg_batch_set_wait_test): one CTA never reaches a barrier, so the
  // others' bounded waits run out and the solve ends with FCG_ERR_TIMEOUT
  if ((int)blockIdx.x == absent_block) return;
  make_split(sp, sys, nsys, true);
  // initial residual res = su - A x, res0 = sum|res|, sk = sum res^2 / a_PP (dpcg.f90:51-90)
  for_share(sp, sys, nsys, spi, [&](int k, int s0, int s1) {
    const double2 t = residual_rows<false>(sys[k], s0, s1);
    double v[2] = {t.x, t.y};
    put_partial<2>(v, part, k, sh);
  });
  if (!grid_sync(ctl, spin_limit, [&] { close_phase(kInit, sys, ctl, sp, nsys, part); })) return;
  int active = nsys;
  for (int loop = 0;; ++loop) {
    const int now = __ldcg(&ctl->nactive);
    if (now <= 0) break;
    if (loop > max_loops) {
      if (blockIdx.x == 0 && threadIdx.x == 0) atomicExch(&ctl->err, 2);
      return;
    }
    if (now != active) make_split(sp, sys, nsys, false);
    active = now;
    // p = a_PP^-1 res + bet p (dpcg.f90:85-100)
    for_share(sp, sys, nsys, spi, [&](int k, int s0, int s1) {
      const BSys &S = sys[k];
      const double bet = __ldcg(&S.bet);
      double *p = S.p;
      const double *res = S.res, *invd = S.invd;
      const int r1 = min(S.n, s1 * 32);
#pragma unroll 4
      for (int r = s0 * 32 + threadIdx.x; r < r1; r += kTPB)
        p[r] = res[r] * __ldg(&invd[r]) + bet * p[r];
    });
    if (!grid_sync(ctl, spin_limit)) return;
    // q = A p, alf = sk / p.q (dpcg.f90:105-121)
    for_share(sp, sys, nsys, spi, [&](int k, int s0, int s1) {
      double v[1] = {spmv_rows(sys[k], s0, s1)};
      put_partial<1>(v, part, k, sh);
    });
    if (!grid_sync(ctl, spin_limit, [&] { close_phase(kSpmv, sys, ctl, sp, nsys, part); })) return;
    // x += alf p, res -= alf q, resl = sum|res|, next sk (dpcg.f90:124-142)
    for_share(sp, sys, nsys, spi, [&](int k, int s0, int s1) {
      const BSys &S = sys[k];
      const double alf = __ldcg(&S.alf);
      double *x = S.x, *res = S.res;
      const double *p = S.p, *q = S.q, *invd = S.invd;
      const int r1 = min(S.n, s1 * 32);
      double v[2] = {0.0, 0.0};
#pragma unroll 4
      for (int r = s0 * 32 + threadIdx.x; r < r1; r += kTPB) {
        x[r] = x[r] + alf * p[r];
        const double rr = res[r] - alf * q[r];
        res[r] = rr;
        v[0] += fabs(rr);
        v[1] += rr * (rr * __ldg(&invd[r]));
      }
      put_partial<2>(v, part, k, sh);
    });
    if (!grid_sync(ctl, spin_limit, [&] { close_phase(kUpdate, sys, ctl, sp, nsys, part); })) return;
  }
  // final FP64 check of every system: ||su - A x||^2, ||su||^2
  make_split(sp, sys, nsys, true);
  for_share(sp, sys, nsys, spi, [&](int k, int s0, int s1) {
    const double2 t = residual_rows<true>(sys[k], s0, s1);
    double v[2] = {t.x, t.y};
    put_partial<2>(v, part, k, sh);
  });
  grid_sync(ctl, spin_limit, [&] { close_phase(kFinal, sys, ctl, sp, nsys, part); });
}

}  // namespace
}  // namespace fcg

using namespace fcg;

struct fcg_batch {
  std::vector<fcg_context *> ctx;
  int device = 0, num_sms = 0, occ = 1;
  cudaStream_t stream = nullptr;
  std::string err;
  int slices_per_item = 8, blocks_per_sm = 1;
  DBuf dsys, dpart, dctl;
  BSys *hsys = nullptr;  // pinned: the graph copies it to the device at every launch
  BCtl *hctl = nullptr;
  int items_for = -1;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int graph_grid = 0, graph_loops = 0;
  long long spin_limit = 1LL << 22;  // polls per barrier wait: over a second
  int absent_block = -1;              // diagnostics: a CTA that skips the barriers
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, loaded = nullptr;
};

namespace {

int bfail(fcg_batch *b, int status, const std::string &msg) {
  if (b) b->err = msg;
  return status;
}

#define B_TRY(b, expr)                                                                    \
  do {                                                                                    \
    cudaError_t _e = (expr);                                                              \
    if (_e != cudaSuccess)                                                                \
      return bfail((b), FCG_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(_e)); \
  } while (0)

void drop_graph(fcg_batch *b) {
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  b->exec = nullptr;
  b->graph = nullptr;
}

// Item counts of `slices_per_item` slices for every system, and room for the partials.
int build_items(fcg_batch *b) {
  if (b->items_for == b->slices_per_item) return FCG_OK;
  for (size_t k = 0; k < b->ctx.size(); ++k)
    b->hsys[k].nitems = (b->ctx[k]->sv.nslices + b->slices_per_item - 1) / b->slices_per_item;
  B_TRY(b, b->dpart.ensure(sizeof(double) * 2 * b->ctx.size() * (size_t)b->num_sms * b->occ));
  b->items_for = b->slices_per_item;
  drop_graph(b);
  return FCG_OK;
}

int grid_size(const fcg_batch *b) { return b->num_sms * std::min(b->blocks_per_sm, b->occ); }

// Enqueues one batched solve on b->stream: inputs of hsys, control block, the kernel.
int enqueue(fcg_batch *b, cudaStream_t st, int grid, int max_loops) {
  const size_t ns = b->ctx.size();
  B_TRY(b, cudaMemcpyAsync(b->dsys.p, b->hsys, sizeof(BSys) * ns, cudaMemcpyHostToDevice, st));
  B_TRY(b, cudaMemcpyAsync(b->dctl.p, b->hctl, sizeof(BCtl), cudaMemcpyHostToDevice, st));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kTPB);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  B_TRY(b, cudaLaunchKernelEx(&cfg, k_batch_dpcg, b->dsys.as<BSys>(),
                              (int)ns, b->slices_per_item, b->dpart.as<double>(),
                              b->dctl.as<BCtl>(), max_loops, b->spin_limit, b->absent_block));
  return FCG_OK;
}

bool graphs_off() {
  const char *e = std::getenv("FCG_NO_GRAPH");
  return e && e[0] == '1';
}

// Runs the batch on the systems already loaded (hsys filled); times it with events.
int run(fcg_batch *b, int max_loops, float *ms) {
  int rc = build_items(b);
  if (rc) return rc;
  const int grid = grid_size(b);
  b->hctl->count = 0;
  b->hctl->gen = 0;
  b->hctl->err = 0;
  b->hctl->nactive = (int)b->ctx.size();
  B_TRY(b, cudaEventRecord(b->ev0, b->stream));
  if (graphs_off()) {
    if ((rc = enqueue(b, b->stream, grid, max_loops))) return rc;
  } else {
    if (!b->exec || b->graph_grid != grid || b->graph_loops != max_loops) {
      drop_graph(b);
      cudaStream_t cap;
      B_TRY(b, cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
      cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
      if (e == cudaSuccess) {
        rc = enqueue(b, cap, grid, max_loops);
        cudaGraph_t g = nullptr;
        e = cudaStreamEndCapture(cap, &g);
        if (!rc && e == cudaSuccess) {
          e = cudaGraphInstantiate(&b->exec, g, 0);
          if (e == cudaSuccess) b->graph = g;
          else cudaGraphDestroy(g);
        } else if (g) {
          cudaGraphDestroy(g);
        }
      }
      cudaStreamDestroy(cap);
      if (rc) return rc;
      if (e != cudaSuccess)
        return bfail(b, FCG_ERR_CUDA, std::string("capture of the batched solve: ") +
                                          cudaGetErrorString(e));
      b->graph_grid = grid;
      b->graph_loops = max_loops;
    }
    B_TRY(b, cudaGraphLaunch(b->exec, b->stream));
  }
  B_TRY(b, cudaEventRecord(b->ev1, b->stream));
  B_TRY(b, cudaMemcpyAsync(b->hsys, b->dsys.p, sizeof(BSys) * b->ctx.size(),
                           cudaMemcpyDeviceToHost, b->stream));
  B_TRY(b, cudaMemcpyAsync(b->hctl, b->dctl.p, sizeof(BCtl), cudaMemcpyDeviceToHost, b->stream));
  B_TRY(b, cudaStreamSynchronize(b->stream));
  if (ms) B_TRY(b, cudaEventElapsedTime(ms, b->ev0, b->ev1));
  if (b->hctl->err == 1)
    return bfail(b, FCG_ERR_TIMEOUT, "a grid-barrier wait of the batched solve gave up");
  if (b->hctl->err == 2)
    return bfail(b, FCG_ERR_TIMEOUT, "batched solve exceeded its loop bound");
  return FCG_OK;
}

// Loads system k (host or device arrays) into its context and fills hsys[k].
int load_system(fcg_batch *b, int k, const double *a, const double *su, const double *fi,
                double sor, int nsw, void **dfi_out, bool *hfi_out) {
  fcg_context *c = b->ctx[k];
  const size_t n1 = sizeof(double) * c->n;
  void *da = nullptr, *dsu, *dfi;
  bool ha, hsu, hfi;
  int rc;
  if (a && (rc = stage_in(c, a, sizeof(double) * c->nnz, 0, true, &da, &ha)))
    return bfail(b, rc, fcg_last_error(c));
  if ((rc = stage_in(c, su, n1, 1, true, &dsu, &hsu))) return bfail(b, rc, fcg_last_error(c));
  if ((rc = stage_in(c, fi, n1, 2, true, &dfi, &hfi))) return bfail(b, rc, fcg_last_error(c));
  BatchVecs v;
  if ((rc = batch_load(c, (const double *)da, (const double *)dsu, (const double *)dfi, &v)))
    return bfail(b, rc, fcg_last_error(c));
  if (c->stream != b->stream) {  // the batch runs after this system's copies
    B_TRY(b, cudaEventRecord(b->loaded, c->stream));
    B_TRY(b, cudaStreamWaitEvent(b->stream, b->loaded, 0));
  }
  BSys &S = b->hsys[k];
  const int nitems = S.nitems;
  std::memset(&S, 0, sizeof S);
  S.nitems = nitems;
  S.sv = c->sv;
  S.n = c->n;
  S.nsw = nsw;
  S.val = v.val;
  S.invd = v.invd;
  S.su = v.su;
  S.x = v.x;
  S.res = v.res;
  S.p = v.p;
  S.q = v.q;
  S.sor = sor;
  S.small = (double)1e-20f;  // modules_allocatable.f90:27
  S.tol = (double)1e-13f;    // dpcg.f90:37
  S.early = 1;
  if (dfi_out) *dfi_out = dfi;
  if (hfi_out) *hfi_out = hfi;
  return FCG_OK;
}

}  // namespace

extern "C" int fcg_batch_destroy(fcg_batch *b);

extern "C" int fcg_batch_create(fcg_context *const *ctxs, int nsys, fcg_batch **out) {
  if (!ctxs || !out || nsys < 1 || nsys > kMaxBatch) return FCG_ERR_ARG;
  *out = nullptr;
  std::set<fcg_context *> seen;
  for (int k = 0; k < nsys; ++k) {
    if (!ctxs[k] || !ctxs[k]->bound || ctxs[k]->device != ctxs[0]->device) return FCG_ERR_ARG;
    if (ctxs[k]->mv.noc) return FCG_ERR_UNSUPPORTED;  // O-C grid cuts: one system at a time
    if (!seen.insert(ctxs[k]).second) return FCG_ERR_ARG;  // systems share solver vectors
  }
  if (cudaSetDevice(ctxs[0]->device) != cudaSuccess) return FCG_ERR_CUDA;
  fcg_batch *b = new fcg_batch();
  b->ctx.assign(ctxs, ctxs + nsys);
  b->device = ctxs[0]->device;
  b->num_sms = ctxs[0]->num_sms;
  b->stream = ctxs[0]->stream;
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_batch_dpcg, kTPB, 0) != cudaSuccess ||
      occ < 1 || cudaMallocHost(&b->hsys, sizeof(BSys) * nsys) != cudaSuccess ||
      cudaMallocHost(&b->hctl, sizeof(BCtl)) != cudaSuccess ||
      b->dsys.ensure(sizeof(BSys) * nsys) != cudaSuccess ||
      b->dctl.ensure(sizeof(BCtl)) != cudaSuccess || cudaEventCreate(&b->ev0) != cudaSuccess ||
      cudaEventCreate(&b->ev1) != cudaSuccess ||
      cudaEventCreateWithFlags(&b->loaded, cudaEventDisableTiming) != cudaSuccess) {
    cudaGetLastError();
    fcg_batch_destroy(b);
    return FCG_ERR_CUDA;
  }
  b->occ = occ;
  // Six slices a warp before another CTA an SM: a barrier's polls and a phase's partial sums
  // cost more with every CTA.  100 sweeps, ms, with 1, 2, 3, 4 and 6 CTAs an SM: one system of
  // 48^3 (2.8 slices a warp) 2.9, 3.0, 3.0, 3.2, 3.8; of 64^3 (6.7) 3.8, 3.5, 3.6, 3.9, 4.7; of
  // 80^3 (13) 5.1, 4.3, 4.2, 4.4, 5.5; of 100^3 (26) 12.5, 8.1, 7.1, 6.9, 7.4.  12 systems of 7.9
  // M cells in all (204) are fastest with six.
  long long slices = 0;
  for (int k = 0; k < nsys; ++k) slices += ctxs[k]->sv.nslices;
  const long long warps = (long long)b->num_sms * kWarps;
  b->blocks_per_sm = (int)std::min<long long>(occ, 1 + slices / (6 * warps));
  std::memset(b->hsys, 0, sizeof(BSys) * nsys);
  if (build_items(b)) {
    fcg_batch_destroy(b);
    return FCG_ERR_CUDA;
  }
  *out = b;
  return FCG_OK;
}

extern "C" int fcg_batch_destroy(fcg_batch *b) {
  if (!b) return FCG_OK;
  cudaSetDevice(b->device);
  if (b->stream) cudaStreamSynchronize(b->stream);
  drop_graph(b);
  if (b->ev0) cudaEventDestroy(b->ev0);
  if (b->ev1) cudaEventDestroy(b->ev1);
  if (b->loaded) cudaEventDestroy(b->loaded);
  if (b->hsys) cudaFreeHost(b->hsys);
  if (b->hctl) cudaFreeHost(b->hctl);
  b->dsys.release();
  b->dpart.release();
  b->dctl.release();
  delete b;
  return FCG_OK;
}

extern "C" const char *fcg_batch_last_error(const fcg_batch *b) {
  return b ? b->err.c_str() : "NULL batch";
}

extern "C" int fcg_batch_set_params(fcg_batch *b, int slices_per_item, int blocks_per_sm) {
  if (!b || slices_per_item < 1 || slices_per_item > 4096 || blocks_per_sm < 1) return FCG_ERR_ARG;
  if (blocks_per_sm > b->occ)
    return bfail(b, FCG_ERR_ARG, "more CTAs per SM than can be resident for a cooperative launch");
  if (b->blocks_per_sm != blocks_per_sm) drop_graph(b);
  b->slices_per_item = slices_per_item;
  b->blocks_per_sm = blocks_per_sm;
  B_TRY(b, cudaSetDevice(b->device));
  return build_items(b);
}

// Diagnostics for the timeout path: the poll limit of every grid-barrier wait and a CTA
// (absent_block >= 0) that returns before the first barrier.  (polls, -1) restores
// normal operation; polls <= 0 restores the default limit.
extern "C" int fcg_batch_set_wait_test(fcg_batch *b, long long polls, int absent_block) {
  if (!b || absent_block < -1) return FCG_ERR_ARG;
  b->spin_limit = polls > 0 ? polls : (1LL << 22);
  b->absent_block = absent_block;
  drop_graph(b);
  return FCG_OK;
}

extern "C" int fcg_batch_get_params(const fcg_batch *b, int *slices_per_item, int *blocks_per_sm,
                                    int *max_blocks_per_sm) {
  if (!b) return FCG_ERR_ARG;
  if (slices_per_item) *slices_per_item = b->slices_per_item;
  if (blocks_per_sm) *blocks_per_sm = b->blocks_per_sm;
  if (max_blocks_per_sm) *max_blocks_per_sm = b->occ;
  return FCG_OK;
}

extern "C" int fcg_batch_dpcg(fcg_batch *b, const double *const *a, const double *const *su,
                              double *const *fi, double sor, int nsw, double *resor,
                              fcg_solve_report *rep) {
  if (!b || !su || !fi || nsw < 0) return FCG_ERR_ARG;
  B_TRY(b, cudaSetDevice(b->device));
  const int ns = (int)b->ctx.size();
  int rc = build_items(b);
  if (rc) return rc;
  std::vector<void *> dfi(ns);
  std::vector<char> hfi(ns);
  for (int k = 0; k < ns; ++k) {
    if (!su[k] || !fi[k]) return bfail(b, FCG_ERR_ARG, "NULL su or fi");
    bool h = false;
    if ((rc = load_system(b, k, a ? a[k] : nullptr, su[k], fi[k], sor, nsw, &dfi[k], &h)))
      return rc;
    hfi[k] = h;
  }
  float ms = 0.f;
  rc = run(b, nsw + 2, &ms);
  if (rc && rc != FCG_ERR_TIMEOUT) return rc;
  const int timeout = rc;
  for (int k = 0; k < ns; ++k) {
    fcg_context *c = b->ctx[k];
    const BSys &S = b->hsys[k];
    const size_t n1 = sizeof(double) * c->n;
    B_TRY(b, cudaMemcpyAsync(dfi[k], S.x, n1, cudaMemcpyDeviceToDevice, c->stream));
    int r2 = stage_out(c, fi[k], dfi[k], n1, hfi[k] != 0);
    if (r2) return bfail(b, r2, fcg_last_error(c));
    if (resor && S.iter > 0) resor[k] = S.res0;  // dpcg.f90:139
    if (rep) {
      rep[k].res0 = S.res0;
      rep[k].resl = S.resl;
      rep[k].iters = S.iter;
      rep[k].converged = S.converged;
      rep[k].l2_rel = S.l2b > 0 ? std::sqrt(S.l2r / S.l2b) : std::sqrt(S.l2r);
      rep[k].seconds = ms * 1e-3;
    }
  }
  for (int k = 0; k < ns; ++k)
    if (k == 0 || b->ctx[k]->stream != b->ctx[k - 1]->stream)
      B_TRY(b, cudaStreamSynchronize(b->ctx[k]->stream));
  if (timeout) return timeout;
  for (int k = 0; k < ns; ++k)
    if (b->hsys[k].status)
      return bfail(b, b->hsys[k].status, "non-finite value in a batched system");
  return FCG_OK;
}

// Times every (slices per item, CTAs per SM) candidate on `sweeps` fixed sweeps of the
// caller's systems (x = 0, sor = 0) and keeps the fastest.  a, su as in fcg_batch_dpcg.
extern "C" int fcg_batch_autotune(fcg_batch *b, const double *const *a, const double *const *su,
                                  int sweeps, double *best_ms) {
  if (!b || !su || sweeps < 1) return FCG_ERR_ARG;
  B_TRY(b, cudaSetDevice(b->device));
  const int ns = (int)b->ctx.size();
  std::vector<DBuf> zeros(ns);
  const int cand_items[] = {4, 8, 16, 32, 64, 128}, cand_bps[] = {1, 2, 4, kResident};
  int best_spi = b->slices_per_item, best_bps = b->blocks_per_sm;
  float best = 1e30f;
  int rc = FCG_OK;
  for (int k = 0; k < ns && !rc; ++k) {
    if (zeros[k].ensure(sizeof(double) * b->ctx[k]->n) != cudaSuccess)
      rc = bfail(b, FCG_ERR_NOMEM, "autotune scratch");
    else if (cudaMemset(zeros[k].p, 0, sizeof(double) * b->ctx[k]->n) != cudaSuccess)
      rc = bfail(b, FCG_ERR_CUDA, "autotune scratch");
  }
  bool loaded = false;
  for (int spi : cand_items) {
    for (int bps : cand_bps) {
      if (rc || bps > b->occ) continue;
      if ((rc = fcg_batch_set_params(b, spi, bps))) break;
      float t = 0.f;
      for (int rep = 0; rep < 2 && !rc; ++rep) {  // first run warms up
        for (int k = 0; k < ns && !rc; ++k)
          rc = load_system(b, k, (a && !loaded) ? a[k] : nullptr, su[k],
                           zeros[k].as<double>(), 0.0, sweeps, nullptr, nullptr);
        loaded = true;
        if (!rc) rc = run(b, sweeps + 2, &t);
      }
      if (!rc && t < best) {
        best = t;
        best_spi = spi;
        best_bps = bps;
      }
    }
    if (rc) break;
  }
  for (DBuf &z : zeros) z.release();
  if (rc) return rc;
  if (best_ms) *best_ms = best;
  return fcg_batch_set_params(b, best_spi, best_bps);
}
