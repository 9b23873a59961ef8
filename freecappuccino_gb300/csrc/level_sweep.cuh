// DIC / DILU sweeps in one launch on any mesh, in level order, in FP64 for the
// single-system solvers (krylov.cu) and FP32 for the multi-RHS ones (multi.cu).
//
// The rows of one level depend only on rows of earlier levels.  The rows stand in level
// order (LevelOrder: every level padded to a multiple of 32 positions), and the
// coefficients, the factor and the result of a sweep in that order too: a warp takes a
// chunk of 32 positions, reads its data coalesced, waits for the values its rows read and
// stores its results as 32 consecutive words.  A result is its own ready flag (a
// signalling-NaN sentinel until it is written).  Rows that follow one another in a level
// mostly read rows that follow one another in the levels before, so a wait polls a few
// sectors of the second-level cache where the natural order polled one per row and entry.
//
// What bounds it: the chain of levels, each a store, a poll and the row's dependent FMAs.
// What a warp needs of its next chunks is therefore loaded while it waits: the chunk it
// works on, the next one's data and the one after's row list are in flight together.
// Chunks are claimed in ascending order and a warp works on its claims in that order, so
// the first unfinished chunk is always being worked on and the waits end; each is bounded.
// The sentinels of one sweep's result are restored by the other sweep.
//
// Measured (GB300): on 93 x 81 x 77 cells less a step (532 k rows, 249 levels) the FP64
// forward and backward sweeps take 179 us each, 0.7 us a level, against about 890 us each
// with warps claiming rows in the natural order; 40 ICCG sweeps 70.9 -> 16.5 ms.  On
// 150 x 140 x 130 cells, us forward: 351, 319, 310, 319 with 1, 2, 4 and 8 blocks an SM.
#pragma once

#include <algorithm>
#include <utility>

#include "wave_sweep.cuh"

namespace fcg {
namespace level {

using wave::Control;
using wave::Word;
using wave::kBackward;
using wave::kFactor;
using wave::kForward;

constexpr int kThreads = 128;
constexpr int kBlocksPerSM = 4;
constexpr int kW = 4;  // entries of a row held in registers; more are read as they come

// Device arrays of the sweeps; every array holds ns systems one after another.
template <class T>
struct Arrays {
  T *fval, *bval;  // coefficients times the row's d, in the order of dep ([32 ptr[chunks]])
  T *fd, *bd;      // factor, rescale d / (d + small) by position
  T *y, *z;        // results by position (sentinels between applications)
};

template <class T>
struct Item {
  int p, off, w;
  T x, s, d;  // d: the backward sweep's factor (PLAIN)
  int dep[kW];
  T v[kW], t[kW];  // t: a_ji of the factor (PLAIN)
};

// One sweep of ns systems: the factor, y = (b - L y) d from `in` (natural order), or
// z = y rescale - (U z) d into `out` (natural order); see wave_sweep.cuh.
// PLAIN as there; its factor takes the CSR values in `in` and their transposes' places.
// `in` holds in_len values a system.
template <class T, int MODE, bool PLAIN>
__global__ void __launch_bounds__(kThreads)
    k_level_sweep(LevelSide lo, LevelSide up, int n, int ns, Arrays<T> A,
                  const T *__restrict__ in, long long in_len, const int *__restrict__ tpos, T *__restrict__ out, int *ctl, int *fail, int *status,
                  const int *done, int spin, int absent) {
  using W = Word<T>;
  constexpr bool BWD = MODE == kBackward, FACTOR = MODE == kFactor;
  if (__ldcg(done) != 0) return;
  const LevelSide &sd = BWD ? up : lo;
  const int lane = threadIdx.x & 31;
  // the forward sweep also goes over the backward one's chunks to restore its sentinels
  const int units = (BWD ? up.chunks : max(lo.chunks, up.chunks)) * ns;
  const long long len = 32LL * sd.chunks, ylen = 32LL * lo.chunks, zlen = 32LL * up.chunks;
  const long long elen = 32LL * sd.entries;
  const T *val = BWD ? A.bval : A.fval, *dd = BWD ? A.bd : A.fd;
  T *res = BWD ? A.z : A.y;
  auto claim = [&]() {
    int c = 0;
    if (lane == 0) {
      c = atomicAdd(&ctl[BWD ? 1 : 0], 1);
      if (c == 0) ctl[BWD ? 0 : 1] = 0;  // the other sweep's counter, which is not running
    }
    return c;  // in lane 0; broadcast when it is needed
  };
  // where a unit's rows and entries stand
  struct Meta {
    int unit, row, off, w, xp;
  };
  auto meta = [&](int unit) {
    Meta m{unit, -1, 0, 0, 0};
    const int c = unit / ns;
    if (unit < units && c < sd.chunks) {
      m.row = sd.row[32 * c + lane];
      m.off = sd.ptr[c];
      m.w = sd.ptr[c + 1] - m.off;
      if (BWD) m.xp = sd.xpos[32 * c + lane];
    }
    return m;
  };
  auto data = [&](const Meta &m, Item<T> &it) {
    const int c = m.unit / ns, s = m.unit - c * ns;
    it.p = 32 * c + lane;
    it.off = m.off;
    it.w = m.w;
    it.x = T(0);
    it.s = T(0);
    it.d = T(0);
#pragma unroll
    for (int e = 0; e < kW; ++e) {
      it.dep[e] = -1;
      it.v[e] = it.t[e] = T(0);
      if (e < m.w) {
        const long long q = 32LL * (m.off + e) + lane;
        it.dep[e] = sd.dep[q];
        it.v[e] = val[s * elen + q];
        if (PLAIN && FACTOR && sd.src[q] >= 0) it.t[e] = in[s * in_len + tpos[sd.src[q]]];
      }
    }
    if (m.row >= 0) {
      it.s = dd[s * len + it.p];
      if (PLAIN && BWD) it.d = A.fd[s * ylen + m.xp];
      if (BWD)
        it.x = A.y[s * ylen + m.xp];
      else if (!FACTOR)
        it.x = in[s * in_len + m.row];
    }
  };
  Meta m0 = meta(__shfl_sync(0xffffffffu, claim(), 0));
  Meta m1 = meta(__shfl_sync(0xffffffffu, claim(), 0));
  Item<T> it;
  data(m0, it);
  int ahead = claim();
  while (m0.unit < units) {
    Item<T> next;
    data(m1, next);
    const Meta m2 = meta(__shfl_sync(0xffffffffu, ahead, 0));
    ahead = claim();
    const int c = m0.unit / ns, s = m0.unit - c * ns;
    if (!BWD && c < up.chunks) A.z[s * zlen + 32 * c + lane] = W::sentinel();
    const T *r = res + s * len;
    bool ok = true;
    T acc = FACTOR ? it.s : PLAIN && !BWD ? it.x : it.x * it.s;
    for (int e0 = 0; e0 < it.w; e0 += kW) {
      if (e0 > 0) {  // rows of more than kW entries
#pragma unroll
        for (int e = 0; e < kW; ++e) {
          const long long q = 32LL * (it.off + e0 + e) + lane;
          it.dep[e] = e0 + e < it.w ? sd.dep[q] : -1;
          it.v[e] = e0 + e < it.w ? val[s * elen + q] : T(0);
          if (PLAIN && FACTOR)
            it.t[e] = e0 + e < it.w && sd.src[q] >= 0 ? in[s * in_len + tpos[sd.src[q]]] : T(0);
        }
      }
      T v[kW];
      for (int polls = 0;; ++polls) {
        bool wait = false;
#pragma unroll
        for (int e = 0; e < kW; ++e) v[e] = it.dep[e] >= 0 ? W::ld(&r[it.dep[e]]) : T(0);
#pragma unroll
        for (int e = 0; e < kW; ++e) wait |= W::sent(v[e]);
        if (!__any_sync(0xffffffffu, wait)) break;
        bool stop = polls > spin;
        if ((polls & 63) == 63) stop |= __any_sync(0xffffffffu, *(volatile int *)&ctl[3] != 0);
        if (stop) {
          ok = !wait;
          break;
        }
      }
#pragma unroll
      for (int e = 0; e < kW; ++e) {
        if (PLAIN && FACTOR)
          acc = W::sub_rounded(acc, it.v[e] * v[e], it.t[e]);
        else
          acc = PLAIN ? W::sub_rounded(acc, it.v[e], v[e]) : W::sub(acc, it.v[e], v[e]);
      }
    }
    if (!ok && atomicExch(&ctl[3], 1) == 0) {
      if (fail) *fail = 1;
      atomicCAS(status, 0, FCG_ERR_TIMEOUT);
    }
    if (m0.row >= 0) {
      if (FACTOR) acc = T(1) / acc;
      if (PLAIN && !FACTOR) acc = acc * (BWD ? it.d : it.s);
      if (BWD || m0.row != absent || FACTOR) W::st(&res[s * len + it.p], acc);
      if (BWD) {
        out[(long long)s * n + m0.row] = acc;
        A.y[s * ylen + m0.xp] = W::sentinel();
      }
    }
    m0 = m1;
    m1 = m2;
    it = next;
  }
}

// The factor's coefficients a_ij^2 (DIC) or a_ij a_ji (DILU) and a_ii from the CSR values.
template <class T, bool PLAIN>
__global__ void k_level_pack_factor(LevelSide lo, int ns, long long nnz,
                                    const int *__restrict__ diag, const int *__restrict__ tpos,
                                    const T *__restrict__ a, int dilu, Arrays<T> A) {
  const long long len = 32LL * lo.chunks, elen = 32LL * lo.entries;
  FCG_GRID_STRIDE(p, len) {
    const int c = (int)(p >> 5), lane = (int)(p & 31), row = lo.row[p];
    for (int e = lo.ptr[c]; e < lo.ptr[c + 1]; ++e) {
      const long long q = 32LL * e + lane;
      const int k = lo.src[q], kt = k >= 0 && dilu ? tpos[k] : k;
      for (int s = 0; s < ns; ++s)
        A.fval[s * elen + q] = k < 0 ? T(0) : PLAIN ? a[s * nnz + k] : a[s * nnz + k] * a[s * nnz + kt];
    }
    for (int s = 0; s < ns; ++s) A.fd[s * len + p] = row >= 0 ? a[s * nnz + diag[row]] : T(0);
  }
}

// The sweeps' coefficients from the CSR values and the factor, which the factor sweep left
// in A.y; a pivot that is not finite is recorded.
template <class T, bool BWD, bool PLAIN>
__global__ void k_level_pack(LevelSide sd, long long ylen, int ns, long long nnz,
                             const T *__restrict__ a, T small, Arrays<T> A, int *status) {
  const long long len = 32LL * sd.chunks, elen = 32LL * sd.entries;
  FCG_GRID_STRIDE(p, len) {
    const int c = (int)(p >> 5), lane = (int)(p & 31), row = sd.row[p];
    for (int s = 0; s < ns; ++s) {
      const T d = row >= 0 ? A.y[s * ylen + (BWD ? sd.xpos[p] : p)] : T(0);
      for (int e = sd.ptr[c]; e < sd.ptr[c + 1]; ++e) {
        const long long q = 32LL * e + lane;
        const int k = sd.src[q];
        (BWD ? A.bval : A.fval)[s * elen + q] = k < 0 ? T(0) : PLAIN ? a[s * nnz + k] : a[s * nnz + k] * d;
      }
      if (BWD)
        A.bd[s * len + p] = row >= 0 ? (PLAIN ? T(1) : d) / (d + small) : T(0);
      else
        A.fd[s * len + p] = d;
      if (!BWD && !isfinite(d)) atomicCAS(status, 0, FCG_ERR_PIVOT);
    }
  }
}

// Sentinels into both results and the control words cleared.
template <class T>
__global__ void k_level_arm(long long ny, T *y, long long nz, T *z, int *ctl) {
  if (blockIdx.x == 0 && threadIdx.x < 4) ctl[threadIdx.x] = 0;
  FCG_GRID_STRIDE(i, ny) y[i] = Word<T>::sentinel();
  FCG_GRID_STRIDE(j, nz) z[j] = Word<T>::sentinel();
}

template <class T>
int allocate(fcg_context *c, int ns, DBuf &buf, Arrays<T> &A) {
  int rc = level_order(c);
  if (rc) return rc;
  const size_t ef = 32 * (size_t)c->order.lo.entries, eb = 32 * (size_t)c->order.up.entries;
  const size_t lf = 32 * (size_t)c->order.lo.chunks, lb = 32 * (size_t)c->order.up.chunks;
  FCG_CUDA_TRY(c, buf.ensure(sizeof(T) * ns * (ef + eb + 2 * lf + 2 * lb)));
  T *p = buf.as<T>();
  for (auto &a : {std::make_pair(&A.fval, ef), std::make_pair(&A.bval, eb),
                  std::make_pair(&A.fd, lf), std::make_pair(&A.bd, lb), std::make_pair(&A.y, lf),
                  std::make_pair(&A.z, lb)}) {
    *a.first = p;
    p += ns * a.second;
  }
  return FCG_OK;
}

template <class T, bool PLAIN = false>
void launch(fcg_context *c, cudaStream_t st, int ns, int mode, const Arrays<T> &A, const T *in,
            T *out, const Control &w, int absent = -1) {
  auto kernel = mode == kForward    ? k_level_sweep<T, kForward, PLAIN>
                : mode == kBackward ? k_level_sweep<T, kBackward, PLAIN>
                                    : k_level_sweep<T, kFactor, wave::kPlainFactor<T, PLAIN>>;
  const long long in_len = mode == kFactor ? c->nnz : c->n;
  kernel<<<c->num_sms * kBlocksPerSM, kThreads, 0, st>>>(c->order.lo, c->order.up, c->n, ns, A, in,
                                                         in_len, c->tpos, out, w.ctl, w.fail, w.status, w.done,
                                                         w.spin, absent);
}

// The factor, the coefficients and armed results: before the first sweep of a solve.
template <class T, bool PLAIN = false>
int start(fcg_context *c, int ns, long long nnz, const T *a, bool dilu, T small,
          const Arrays<T> &A, const Control &solver) {
  const Control w = solver.unstopped();
  const LevelSide &lo = c->order.lo, &up = c->order.up;
  const long long lf = 32LL * lo.chunks, lb = 32LL * up.chunks;
  const int gf = grid_for(lf, c->num_sms), gb = grid_for(lb, c->num_sms);
  const int ga = grid_for(ns * std::max(lf, lb), c->num_sms);
  constexpr bool PF = wave::kPlainFactor<T, PLAIN>;
  k_level_pack_factor<T, PF><<<gf, kTPB, 0, c->stream>>>(lo, ns, nnz, c->mv.diag, c->tpos, a, dilu, A);
  k_level_arm<T><<<ga, kTPB, 0, c->stream>>>(ns * lf, A.y, ns * lb, A.z, w.ctl);
  launch<T, PLAIN>(c, c->stream, ns, kFactor, A, PF ? a : nullptr, nullptr, w);
  k_level_pack<T, false, PLAIN><<<gf, kTPB, 0, c->stream>>>(lo, lf, ns, nnz, a, small, A, w.status);
  k_level_pack<T, true, PLAIN><<<gb, kTPB, 0, c->stream>>>(up, lf, ns, nnz, a, small, A, w.status);
  k_level_arm<T><<<ga, kTPB, 0, c->stream>>>(ns * lf, A.y, ns * lb, A.z, w.ctl);
  FCG_CHECK_LAUNCH(c, "level-order factor and coefficients");
  return FCG_OK;
}

}  // namespace level
}  // namespace fcg
