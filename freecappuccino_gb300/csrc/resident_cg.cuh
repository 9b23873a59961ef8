// DPCG on a system that the resident threads hold: the whole iteration in one cooperative
// launch.  Included by krylov.cu.
//
// Every thread keeps kRows rows' x, residual and direction in registers.  A sweep is two
// phases, each closed by a grid-wide sum: q = A p with p.q, and the update with sum|res| and
// the next sk.  The direction needs no phase of its own: a row forms its neighbours' new
// directions z + bet p_old as it reads them (z = res / a_PP is the update's; both vectors
// are double-buffered).
//
// What bounds it: the latency of the two sums, 7 us each: a store and a poll through L2, and
// some 40 dependent FP64 instructions (additions of lanes, warps and blocks, the quotients)
// of 64 issue cycles.  The captured loop's three kernels take 32 us a sweep at any size below
// 110 k rows, nearly all of it launches and tickets; this takes 14 at 14 k and 33 k rows, 21
// at 110 k and 31 at 300 k (the loop: 42).  A system past four rows a thread goes to the
// loop, which streams its vectors as fast as the FP64 pipe allows.
#pragma once

namespace fcg {
namespace {

constexpr int kResidentThreads = 512;  // a block's largest size; one block an SM
constexpr int kResidentBlocks = 160;   // at most
constexpr int kResidentRows = 4;       // rows a thread, at most

constexpr int kResidentPolls = 1 << 21;  // of a wait before it gives up: over a second

// Doubles of one set of slots of G blocks: even, so that pairs are aligned.
__host__ __device__ constexpr int slot_set(int G) { return (G * G + 1) & ~1; }

struct ResidentCg {
  SellView s;
  int n;
  const double *val, *invd;
  double *x, *res, *z0, *z1, *p0, *p1;  // p0: the direction on return (zero before)
  Scal *S;
  double *slots;  // five sets (grid_sums)
  double *trace;
  int polls;    // of a wait before it gives up
  int quitter;  // diagnostics (fcg_set_sweep_wait_test): the block whose first wait for the
                // update's sums counts as given up; -1: none
};

// A slot that is not written yet: a signalling NaN, which no sum of doubles results in.
constexpr unsigned long long kEmpty = 0x7ff4dead7ff4deadULL;

// What the first sweep reads: empty slots and z = res / a_PP.
__global__ void __launch_bounds__(kTPB) k_resident_start(ResidentCg a, int blocks) {
  FCG_GRID_STRIDE(i, 5 * slot_set(blocks)) a.slots[i] = __longlong_as_double(kEmpty);
  FCG_GRID_STRIDE(r, a.n) a.z0[r] = __dmul_rn(a.res[r], a.invd[r]);
}

// Grid-wide sums of v, handed to close(v), which one thread of every block runs; what close
// wrote to shared memory is visible to the block after it.  False: a wait gave up.
//
// A sweep sums twice: A, p.q, and B, sum|res| and the next sk.  Every block writes its
// partial sum into a slot of every block, so that a block polls lines that no other block
// polls (all blocks on the same slots: 23 us a sweep at 24^3, against 15).  A block
// empties its slots as it reads them.  Only B is fenced: what a block writes before a B is
// visible to all after it, which is when the others write the next A's slots; B's slots are
// used in two sets in turn, so that an emptied set has passed a fenced B too.
template <int NV>
__device__ __forceinline__ void slot_write(double *slot, const double *v) {
  if (NV == 1)
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(slot), "d"(v[0]) : "memory");
  else
    asm volatile("st.volatile.global.v2.f64 [%0], {%1, %2};" ::"l"(slot), "d"(v[0]), "d"(v[NV - 1])
                 : "memory");
}

template <int NV>
__device__ __forceinline__ void slot_read(const double *slot, double *v) {
  if (NV == 1)
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v[0]) : "l"(slot) : "memory");
  else
    asm volatile("ld.volatile.global.v2.f64 {%0, %1}, [%2];"
                 : "=d"(v[0]), "=d"(v[NV - 1])
                 : "l"(slot)
                 : "memory");
}

// Sums of v over the first `span` lanes (a power of two; the rest hold zero), in every lane.
// Two values cost the additions of one and a half: after the first exchange each half of the
// lanes carries one of them.  An FP64 addition issues for 64 cycles.
template <int NV>
__device__ __forceinline__ void lane_sums(double (&v)[NV], int span) {
  if (NV == 1) {
    for (int o = span >> 1; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    v[0] = __shfl_sync(0xffffffffu, v[0], 0);
  } else {
    const bool high = threadIdx.x & 16;
    const double give = high ? v[0] : v[NV - 1], keep = high ? v[NV - 1] : v[0];
    double t = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    for (int o = min(span, 16) >> 1; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    v[0] = __shfl_sync(0xffffffffu, t, 0);
    v[NV - 1] = __shfl_sync(0xffffffffu, t, 16);
  }
}

template <int NV, class F>
__device__ __forceinline__ bool grid_sums(const ResidentCg &a, int sweep, double (&v)[NV],
                                          double (*sh)[kResidentThreads / 32], int *failed,
                                          F &&close) {
  const int G = gridDim.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
  constexpr int M = kResidentBlocks / 32;
  lane_sums<NV>(v, 32);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[k][w] = v[k];
  __syncthreads();
  if (w == 0) {
    // [reader][writer][NV]: one set of A, then two of B
    const int set = slot_set(G);
    double *slots = a.slots + (NV == 1 ? 0 : set + (sweep & 1) * 2 * set);
    double *mine = slots + (long long)blockIdx.x * G * NV;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = lane < W ? sh[k][lane] : 0.0;
    if (NV == 2) __threadfence();
    lane_sums<NV>(v, W > 8 ? 16 : W > 4 ? 8 : W > 2 ? 4 : W);
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int reader = lane + 32 * m;
      if (reader < G) slot_write<NV>(slots + ((long long)reader * G + blockIdx.x) * NV, v);
    }
    // all of a lane's slots are read together, again until none is empty
    double t[M][NV];
    int left = a.polls;
    bool wait;
    do {
      wait = false;
#pragma unroll
      for (int m = 0; m < M; ++m) {
#pragma unroll
        for (int k = 0; k < NV; ++k) t[m][k] = 0.0;
        if (lane + 32 * m < G) slot_read<NV>(mine + (lane + 32 * m) * NV, t[m]);
      }
#pragma unroll
      for (int m = 0; m < M; ++m)
#pragma unroll
        for (int k = 0; k < NV; ++k) wait |= __double_as_longlong(t[m][k]) == kEmpty;
    } while (wait && --left > 0);
    if (NV == 2 && (int)blockIdx.x == a.quitter) wait = true;
#pragma unroll
    for (int m = 0; m < M; ++m)
      if (lane + 32 * m < G) {
        const double e = __longlong_as_double(kEmpty), none[2] = {e, e};
        slot_write<NV>(mine + (lane + 32 * m) * NV, none);
      }
    const bool ok = !__any_sync(0xffffffffu, wait);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      v[k] = t[0][k];
#pragma unroll
      for (int m = 1; m < M; ++m)
        if (32 * m < G) v[k] += t[m][k];
    }
    lane_sums<NV>(v, 32);
    if (lane == 0) {
      if (ok) {
        close(v);
      } else {
        *failed = 1;
        a.S->wait_fail = 2;
        fail_status(a.S, FCG_ERR_TIMEOUT);
      }
    }
    if (NV == 2) __threadfence();
  }
  __syncthreads();
  return !*(volatile int *)failed;
}

// acc = sum a_j (z + bet p)[c_j], in slot order; the vectors are other blocks' writes
template <int BATCH>
__device__ __forceinline__ double direction_row(const ResidentCg &a, const double *z,
                                                const double *p, double bet, int slice,
                                                int lane) {
  const long long base = __ldg(&a.s.ptr[slice]) + lane;
  const int w = __ldg(&a.s.width[slice]), op = __ldg(&a.s.offp[slice]);
  const bool uniform = __ldg(&a.s.kind[slice]) == 0;
  const int row = slice * 32 + lane;
  double acc = 0.0;
  for (int j0 = 0; j0 < w; j0 += BATCH) {
    double v[BATCH], zc[BATCH], pc[BATCH];
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      v[u] = zc[u] = pc[u] = 0.0;
      if (j0 + u < w) {
        int c = uniform ? row + __ldg(&a.s.off[op + j0 + u])
                        : __ldg(&a.s.off[op + 32 * (j0 + u) + lane]);
        c = c < 0 ? 0 : (c >= a.n ? a.n - 1 : c);
        v[u] = __ldg(&a.val[base + (long long)(j0 + u) * 32]);
        zc[u] = __ldcg(&z[c]);
        pc[u] = __ldcg(&p[c]);
      }
    }
#pragma unroll
    for (int u = 0; u < BATCH; ++u)
      if (j0 + u < w) acc += v[u] * fma(bet, pc[u], zc[u]);
  }
  return acc;
}

template <int R>
__global__ void __launch_bounds__(kResidentThreads, 1) k_resident_dpcg(ResidentCg a) {
  __shared__ Scal sc;  // the block's copy of the scalars; block 0 returns the solve's
  __shared__ double sh[2][kResidentThreads / 32];
  __shared__ int failed;
  if (solve_done(a.S)) return;
  if (threadIdx.x == 0) {
    sc = *a.S;
    failed = 0;
  }
  const int lane = threadIdx.x & 31, W = blockDim.x >> 5;
  const int first = blockIdx.x * W + (threadIdx.x >> 5), step = gridDim.x * W;
  double x[R], res[R], p[R], invd[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = (first + i * step) * 32 + lane;
    x[i] = res[i] = p[i] = invd[i] = 0.0;
    if (r < a.n) {
      x[i] = a.x[r];
      res[i] = a.res[r];
      invd[i] = a.invd[r];
    }
  }
  __syncthreads();
  const int nsw = sc.nsw;
  // sweep s reads directions p[s % 2] and residuals z[s % 2] and writes the others
  for (int it = 0; it < nsw; ++it) {
    const double *pold = it & 1 ? a.p1 : a.p0, *z = it & 1 ? a.z1 : a.z0;
    double *pnew = it & 1 ? a.p0 : a.p1, *znew = it & 1 ? a.z0 : a.z1;
    double q[R], v[1] = {0.0};
    const double bet = sc.bet;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int slice = first + i * step, r = slice * 32 + lane;
      q[i] = 0.0;
      if (slice < a.s.nslices) {
        q[i] = direction_row<R == 1 ? 8 : 4>(a, z, pold, bet, slice, lane);
        if (r < a.n) {
          p[i] = fma(bet, p[i], __dmul_rn(res[i], invd[i]));  // as its neighbours form it
          pnew[r] = p[i];
          v[0] += p[i] * q[i];
        }
      }
    }
    if (!grid_sums<1>(a, it, v, sh, &failed, [&](double *t) {
          sc.pkapk = t[0];
          sc.alf = sc.sk / t[0];
          if (!isfinite(sc.alf)) fail_status(&sc, FCG_ERR_NONFINITE);
        }))
      return;
    const double alf = sc.alf;
    double t[2] = {0.0, 0.0};
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = (first + i * step) * 32 + lane;
      if (r < a.n) {
        x[i] = x[i] + alf * p[i];
        res[i] = res[i] - alf * q[i];
        const double zr = __dmul_rn(res[i], invd[i]);
        znew[r] = zr;
        t[0] += fabs(res[i]);
        t[1] += res[i] * zr;
      }
    }
    if (!grid_sums<2>(a, it, t, sh, &failed, [&](double *u) {
          cg_close_sweep(&sc, u[0], u[1], blockIdx.x == 0 ? a.trace : nullptr, 0, 0, SK_DPCG);
        }))
      return;
    if (sc.done) break;
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = (first + i * step) * 32 + lane;
    if (r < a.n) {
      a.x[r] = x[i];
      a.res[r] = res[i];
      a.p0[r] = p[i];
    }
  }
  // Only what the sweeps change, and a status of this block's beside one that is there:
  // another block may have given up on the last sums, which this one saw complete, and left
  // without storing its rows.
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    Scal *S = a.S;
    S->resl = sc.resl;
    S->resor = sc.resor;
    S->rsm = sc.rsm;
    S->s0 = sc.s0;
    S->sk = sc.sk;
    S->bet = sc.bet;
    S->pkapk = sc.pkapk;
    S->alf = sc.alf;
    S->iter = sc.iter;
    S->done = sc.done;
    S->converged = sc.converged;
    if (sc.status) fail_status(S, sc.status);
  }
}

}  // namespace
}  // namespace fcg
