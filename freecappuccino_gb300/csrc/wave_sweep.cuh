// Wavefront-tiled DIC / DILU sweeps on a lexicographic hex block (c->hex), in FP64 for
// the single-system solvers (krylov.cu) and FP32 for the multi-RHS ones (multi.cu).
//
// The cells form an nx x ny x nz block; the lower entries of row r are (when present, in CSR
// order) r - nx ny, r - nx, r - 1 and the upper ones r + 1, r + nx, r + nx ny.  A block of
// TX x TY threads owns a tile of (i, j) columns and walks it in wavefront order: at step L
// the thread of column (di, dj) of the tile computes the cell k = L - di - dj (the
// backward sweep takes the steps in descending order).  The cell's upstream neighbour in k
// is the thread's own previous cell (a register); those in i and j inside the tile were
// computed one step earlier by the neighbouring threads (shared memory, double buffered,
// one barrier a step).
//
// The tile's first (backward: last) row and column read cells of another tile.  They take
// them from an edge buffer in the tile's shared memory, filled with a signalling-NaN
// sentinel at the start; a value that is still the sentinel is polled there (bounded):
//   - CX x CY tiles form a thread-block cluster, whose blocks store their edge results
//     straight into the neighbour's buffer (distributed shared memory);
//   - across clusters the results go through global memory, also sentinel-armed, and one
//     more warp of the reading block polls there and copies into the buffer.
// Clusters are claimed through an atomic counter in an order in which a cluster's upstream
// clusters come first, so a block only waits for blocks that are running.
//
// What bounds it: the chain of 3N - 2 dependent steps and the hand-over from tile to tile.
// A step is three dependent FMAs (about 88 cycles each in FP64 on this part, which also
// hold the issue of an SM quarter for 64): the own column's before the barrier, the two
// in-tile neighbours' after it.  Everything else is kept off the chain:
//   - the scaling by the factor is folded into the coefficients (a d) and the input (b d);
//   - coefficients, factor, rescale and the forward result are stored in wavefront order
//     (Layout: for every tile and step, TX x TY consecutive values), so that a step's
//     loads are one pointer plus constant offsets, coalesced, and issued kD steps ahead
//     into a register ring whose slots are compile-time constants;
//   - cells outside the block have coefficient, factor and input 0 and compute 0;
//   - the global sentinels are restored by the other sweep (the backward sweep re-arms the
//     forward result it reads, the forward sweep the backward one's edges), so no fill
//     runs between sweeps.
// A hand-over through global memory costs 4-6 us with the tiles spread over the two dies
// (store, second-level cache, poll), one through distributed shared memory well below 1.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "fcg_internal.h"
#include "launch.h"

namespace fcg {
namespace wave {

constexpr int TX = 16, TY = 8, NT = TX * TY;  // columns of a tile, one thread each
constexpr int CX = 2, CY = 4;                 // tiles of a cluster
constexpr int kThreads = NT + 32;             // and the warp that polls for other clusters
constexpr int kD = 8;     // steps that a cell's inputs are loaded ahead
constexpr int kPlanes = 4;
constexpr int kSlab = 512;  // planes of one launch: the edge buffers' length

template <class T>
struct Word;
template <>
struct Word<double> {
  using U = unsigned long long;
  static constexpr U kSent = 0x7ff0dead0badf00dULL;
  static __device__ __forceinline__ double ld(const double *p) {
    U v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return __longlong_as_double((long long)v);
  }
  static __device__ __forceinline__ void st(double *p, double x) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p),
                 "l"((U)__double_as_longlong(x))
                 : "memory");
  }
  // into the shared memory of another block of the cluster
  static __device__ __forceinline__ void push(uint32_t p, double x) {
    asm volatile("st.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(p),
                 "l"((U)__double_as_longlong(x))
                 : "memory");
  }
  static __device__ __forceinline__ double peek(uint32_t p) {
    U v;
    asm volatile("ld.relaxed.cluster.shared::cta.b64 %0, [%1];" : "=l"(v) : "r"(p) : "memory");
    return __longlong_as_double((long long)v);
  }
  // the upper half alone tells: arithmetic gives quiet NaNs only
  static __device__ __forceinline__ bool sent(double v) {
    return (unsigned)__double2hiint(v) == (unsigned)(kSent >> 32);
  }
  static __device__ __forceinline__ double sentinel() {
    return __longlong_as_double((long long)kSent);
  }
  // acc - a v, the product not rounded on its own
  static __device__ __forceinline__ double sub(double acc, double a, double v) {
    return __fma_rn(-a, v, acc);
  }
  // ... and rounded
  static __device__ __forceinline__ double sub_rounded(double acc, double a, double v) {
    return __dsub_rn(acc, __dmul_rn(a, v));
  }
};
template <>
struct Word<float> {
  using U = unsigned;
  static constexpr U kSent = 0x7f80deadu;
  static __device__ __forceinline__ float ld(const float *p) {
    U v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return __uint_as_float(v);
  }
  static __device__ __forceinline__ void st(float *p, float x) {
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(__float_as_uint(x))
                 : "memory");
  }
  static __device__ __forceinline__ void push(uint32_t p, float x) {
    asm volatile("st.relaxed.cluster.shared::cluster.b32 [%0], %1;" ::"r"(p),
                 "r"(__float_as_uint(x))
                 : "memory");
  }
  static __device__ __forceinline__ float peek(uint32_t p) {
    U v;
    asm volatile("ld.relaxed.cluster.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
    return __uint_as_float(v);
  }
  static __device__ __forceinline__ bool sent(float v) { return __float_as_uint(v) == kSent; }
  static __device__ __forceinline__ float sentinel() { return __uint_as_float(kSent); }
  static __device__ __forceinline__ float sub(float acc, float a, float v) {
    return __fmaf_rn(-a, v, acc);
  }
  static __device__ __forceinline__ float sub_rounded(float acc, float a, float v) {
    return __fsub_rn(acc, __fmul_rn(a, v));
  }
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// The address of the same shared-memory location in block `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_addr(uint32_t p, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(p), "r"(rank));
  return r;
}

// Wavefront order of one system: cell (i, j, k) of column (di, dj) of tile t stands at
// (t nlev + L) NT + dj TX + di with L = k + di + dj.
struct Layout {
  int nx, ny, nz, ntx, nty, nsx, nsy, nlev;
  __host__ __device__ Layout(int nx_, int ny_, int nz_)
      : nx(nx_), ny(ny_), nz(nz_), ntx((nx_ + TX - 1) / TX), nty((ny_ + TY - 1) / TY),
        nsx((ntx + CX - 1) / CX), nsy((nty + CY - 1) / CY), nlev(nz_ + TX + TY - 2) {}
  __host__ __device__ int clusters() const { return nsx * nsy; }
  __host__ __device__ long long len() const { return (long long)ntx * nty * nlev * NT; }
  __host__ __device__ long long at(int i, int j, int k) const {
    const long long t = (long long)(j / TY) * ntx + i / TX;
    return (t * nlev + k + i % TX + j % TY) * NT + (j % TY) * TX + i % TX;
  }
  // Lengths of the records and of the vectors of one system.  The guards: the ring loads
  // up to kD steps past the last (backward: before the first) step without a test.
  __host__ __device__ static constexpr long long guard() { return (long long)kD * kPlanes * NT; }
  __host__ __device__ long long rec_len() const { return kPlanes * len() + 2 * guard(); }
  __host__ __device__ long long vec_len() const { return len() + 2 * guard(); }
};

// Device arrays of the sweeps (system s at s times the length above); the pointers are
// past the first guard.  The record of step L of tile t starts at (t nlev + L) kPlanes NT:
// forward planes {lower k, lower j, lower i, factor d}, backward {upper i, upper j,
// upper k, rescale}, the coefficients times the row's d.
template <class T>
struct Arrays {
  T *fwd, *bwd;
  T *y;   // forward result, wavefront order (sentinel on the last rows and columns between
          // applications)
  T *ze;  // backward result on the tiles' first rows and columns (likewise)
};

constexpr int kForward = 0, kBackward = 1, kFactor = 2;

// One sweep of ns systems over the planes [k0, k1): the factor y = 1/(a_ii - sum w y) from
// the forward records {w of lower k, lower j, lower i, a_ii} (w = a_ij^2 for DIC, a_ij a_ji
// for DILU), forward y = (b - L y) d from `in`
// (natural order, system s at s n), or backward z = y rescale - (U z) d into `out`
// (natural order), rescale = d / (d + small).
// Measured (GB300, FP64, us forward / backward): 128^3 143 / 153 against 356 / 380 with the
// coefficients read in natural order through address arithmetic and validity tests, the
// scaling on the chain and every hand-over through global memory; 40 ICCG sweeps at 128^3
// 34.7 -> 16.0 ms, at 256^3 125 -> 60 ms.  One tile alone takes 0.28 us a step (FP32 0.16).
// kD = 4 or 12 measured 189 and 170 us forward at 128^3 and 1217 and 475 us at 256^3
// (kD = 8: 156 and 473); clusters of 1 x 8, 4 x 2 or 4 x 4 tiles are within 3% of 2 x 4.
//
// PLAIN: every operation of a row rounded on its own, in the reference's form: the factor
// a_ii - (a_ij y) a_ji (the a_ji in the backward records), y = (b - L y) d and
// z = (y / (d + small) - U z) d with unscaled coefficients.  For BiCGStab, whose iterates on
// a pressure system magnify an ulp by ten orders of magnitude in 50 sweeps.  Two operations
// a neighbour instead of one and the scaling on the chain: 191 / 223 us at 128^3.  The FP32
// factor is the PLAIN one whatever the sweeps: a_ij a_ji leaves FP32's range for coefficients
// above 1.8e19 or below 1e-19, (a_ij y) a_ji does not.
template <class T, int MODE, bool PLAIN>
__global__ void __launch_bounds__(kThreads) __cluster_dims__(CX *CY, 1, 1)
    k_wave_sweep(int nx, int ny, int nz, int k0, int k1, int ns, Arrays<T> A,
                 const T *__restrict__ in, T *out, int *ctl, int *fail, int *status,
                 const int *done, int spin, int absent) {
  using W = Word<T>;
  constexpr int P = kPlanes;
  constexpr bool BWD = MODE == kBackward, FACTOR = MODE == kFactor;
  if (__ldcg(done) != 0) return;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char wave_smem[];
  __shared__ T sm[kD][TY][TX];
  __shared__ int claim;
  const int depth = k1 - k0;
  T *ebuf = reinterpret_cast<T *>(wave_smem);  // [TY] rows of i edges, [TX] rows of j edges
  const Layout lay(nx, ny, nz);
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x;
  if (rank == 0 && tid == 0) {
    claim = atomicAdd(&ctl[BWD ? 1 : 0], 1);
    if (claim == 0) ctl[BWD ? 0 : 1] = 0;  // the other sweep's counter, which is not running
  }
  // Another block's shared memory may be touched only once every block of the cluster has
  // started, so the claim is read after this barrier, not handed out before it.  Rank 0 leaves
  // after the last cluster.sync() below, its copy is there as long as it is read.
  cluster.sync();
  int claimed;
  asm volatile("ld.shared::cluster.b32 %0, [%1];"
               : "=r"(claimed)
               : "r"(peer_addr(smem_addr(&claim), 0))
               : "memory");
  const int c = claimed / ns, sys = claimed - c * ns;
  const int sc = BWD ? lay.clusters() - 1 - c : c;
  const int cx = rank % CX, cy = rank / CX;
  const int ti = (sc % lay.nsx) * CX + cx, tj = (sc / lay.nsx) * CY + cy;
  const bool tile_ok = ti < lay.ntx && tj < lay.nty;
  // the upstream tiles: none (an edge of zeros), in this cluster, or in another one
  const bool has_p = tile_ok && (BWD ? ti < lay.ntx - 1 : ti > 0);
  const bool has_q = tile_ok && (BWD ? tj < lay.nty - 1 : tj > 0);
  const bool far_p = has_p && (BWD ? cx == CX - 1 : cx == 0);
  const bool far_q = has_q && (BWD ? cy == CY - 1 : cy == 0);
  for (int e = tid; e < TY * depth; e += kThreads) ebuf[e] = has_p ? W::sentinel() : T(0);
  for (int e = tid; e < TX * depth; e += kThreads)
    ebuf[TY * depth + e] = has_q ? W::sentinel() : T(0);
  if (tid < NT) sm[0][tid / TX][tid % TX] = T(0);
  cluster.sync();  // every buffer is armed before any neighbour stores into it
  const int nlev = lay.nlev;
  const long long vl = lay.vec_len();
  const long long tile0 = ((long long)tj * lay.ntx + ti) * nlev * NT;
  const T *E = (BWD ? A.ze : A.y) + sys * vl;  // where other clusters leave their edges
  if (tile_ok && tid >= NT) {
    // the polling warp: lane e < TY takes i-edge row e, the next TX lanes the j-edge rows
    const int e = tid - NT;
    const bool is_p = e < TY;
    const int row = is_p ? e : e - TY;
    const bool mine = e < TY + TX && (is_p ? far_p : far_q);
    T *dst = ebuf + (is_p ? row : TY + row) * depth;
    // cell k of the upstream tile's last (backward: first) column at that row
    const long long nb = BWD ? (is_p ? 1LL : (long long)lay.ntx) : (is_p ? -1LL : -(long long)lay.ntx);
    const int ndi = is_p ? (BWD ? 0 : TX - 1) : row, ndj = is_p ? row : (BWD ? 0 : TY - 1);
    // diagnostics: what this column leaves for other clusters never arrives
    const int from = is_p ? ti * TX - 1 + nx * (tj * TY + row) : ti * TX + row + nx * (tj * TY - 1);
    const bool lost = MODE == kForward && from == absent;
    const T *src = E + tile0 + nb * nlev * NT + (long long)(ndi + ndj) * NT + ndj * TX + ndi;
    constexpr int B = 8;  // cells asked for together
    int at = 0, idle = 0;
    while (__any_sync(0xffffffffu, mine && at < depth)) {
      T v[B];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        v[u] = W::sentinel();
        if (mine && !lost && at + u < depth) {
          const int k = BWD ? k1 - 1 - at - u : k0 + at + u;
          v[u] = W::ld(src + (long long)k * NT);
        }
      }
      int got = 0;
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (got == u && !W::sent(v[u])) {
          const int k = BWD ? k1 - 1 - at - u : k0 + at + u;
          *(volatile T *)(dst + (k - k0)) = v[u];
          ++got;
        }
      at += got;
      // bounded: give up after `spin` rounds without progress of the warp, or when another
      // wait has given up
      idle = __any_sync(0xffffffffu, got > 0) ? 0 : idle + 1;
      if (idle > spin || ((idle & 63) == 63 && *(volatile int *)&ctl[3])) {
        if ((tid & 31) == 0 && atomicExch(&ctl[3], 1) == 0) {
          if (fail) *fail = 1;
          atomicCAS(status, 0, FCG_ERR_TIMEOUT);
        }
        break;
      }
    }
  } else if (tile_ok) {
    const int di = tid % TX, dj = tid / TX;
    const int i = ti * TX + di, j = tj * TY + dj;
    const bool col_ok = i < nx && j < ny;
    const int nxy = nx * ny;
    const long long n = (long long)nxy * nz;
    constexpr int step = BWD ? -1 : 1;
    const int L0 = BWD ? k1 - 1 + TX + TY - 2 : k0;
    // Everything below stands at the first step of a round of kD; a round's accesses are
    // constant offsets from it.
    int k = L0 - di - dj - k0;  // the cell, counted from the slab's first plane
    const T *rec = (BWD ? A.bwd : A.fwd) + sys * lay.rec_len() + (tile0 + (long long)L0 * NT) * P +
                   tid;
    T *yw = A.y + sys * vl + tile0 + (long long)L0 * NT + tid;
    T *zw = A.ze + sys * vl + tile0 + (long long)L0 * NT + tid;
    // natural position of the column's cell, from the slab's first plane on
    const T *xin = MODE != kForward ? nullptr : in + i + (long long)nx * j + (long long)nxy * k0 + sys * n;
    T *xout = BWD ? out + i + (long long)nx * j + (long long)nxy * k0 + sys * n : nullptr;
    // The neighbours' values of step u stand at p_at + u p_inc and q_at + u q_inc: for the
    // tile's first (last) row and column in the edge buffers, cell by cell; for the others
    // in slot u of the tile's results (step u writes slot u + 1, modulo kD).
    const bool edge_p = BWD ? di == TX - 1 : di == 0, edge_q = BWD ? dj == TY - 1 : dj == 0;
    constexpr uint32_t slot = sizeof(T) * NT;
    uint32_t p_at = edge_p ? smem_addr(ebuf + dj * depth) + (uint32_t)(k * (int)sizeof(T))
                           : smem_addr(&sm[0][dj][di - step]);
    uint32_t q_at = edge_q ? smem_addr(ebuf + (TY + di) * depth) + (uint32_t)(k * (int)sizeof(T))
                           : smem_addr(&sm[0][dj - step][di]);
    const uint32_t p_inc = edge_p ? (uint32_t)(step * (int)sizeof(T)) : slot;
    const uint32_t q_inc = edge_q ? (uint32_t)(step * (int)sizeof(T)) : slot;
    const uint32_t p_round = edge_p ? kD * p_inc : 0u, q_round = edge_q ? kD * q_inc : 0u;
    // downstream tiles: in this cluster (store into their buffer) or in another one (the
    // forward result is stored globally anyway, the backward one into ze)
    const bool out_p = BWD ? di == 0 && ti > 0 : di == TX - 1 && ti < lay.ntx - 1;
    const bool out_q = BWD ? dj == 0 && tj > 0 : dj == TY - 1 && tj < lay.nty - 1;
    const bool near_p = out_p && (BWD ? cx > 0 : cx < CX - 1);
    const bool near_q = out_q && (BWD ? cy > 0 : cy < CY - 1);
    const bool far_out = (out_p && !near_p) || (out_q && !near_q);
    const bool rearm_y = di == TX - 1 || dj == TY - 1, rearm_z = di == 0 || dj == 0;
    uint32_t push_p = peer_addr(smem_addr(ebuf + dj * depth), near_p ? rank + step : rank) +
                      (uint32_t)(k * (int)sizeof(T));
    uint32_t push_q = peer_addr(smem_addr(ebuf + (TY + di) * depth), near_q ? rank + step * CX : rank) +
                      (uint32_t)(k * (int)sizeof(T));
    struct Cell {
      T c[P], x;
      T e[PLAIN ? (FACTOR ? 3 : 1) : 1];  // PLAIN: factor a_ji, backward d
    };
    const long long other = FACTOR ? A.bwd - A.fwd : A.fwd - A.bwd;  // to the other record
    auto sub = [](T acc, T a, T v) {
      return PLAIN ? W::sub_rounded(acc, a, v) : W::sub(acc, a, v);
    };
    // acc less the factor's term of neighbour q
    auto term = [&](T acc, const Cell &cl, int q, T v) {
      if constexpr (PLAIN && FACTOR) return W::sub_rounded(acc, cl.c[q] * v, cl.e[q]);
      return sub(acc, cl.c[q], v);
    };
    Cell ring[kD];
    // The inputs of step u (of this round or, from kD on, the next).  Only loads: an
    // instruction that used a loaded value would hold the warp's issue.
    auto load = [&](int u, Cell &cl) {
#pragma unroll
      for (int p = 0; p < P; ++p) cl.c[p] = __ldg(rec + step * u * (P * NT) + p * NT);
      if constexpr (PLAIN && FACTOR) {
#pragma unroll
        for (int p = 0; p < 3; ++p) cl.e[p] = __ldg(rec + other + step * u * (P * NT) + p * NT);
      } else if constexpr (PLAIN && BWD) {
        cl.e[0] = __ldg(rec + other + step * u * (P * NT) + 3 * NT);
      }
      if (BWD) {
        cl.x = yw[step * u * NT];
      } else if (!FACTOR) {
        const int kk = k + u;
        cl.x = T(0);
        if ((unsigned)kk < (unsigned)depth && col_ok) cl.x = __ldg(xin + (long long)nxy * kk);
      }
    };
    // the part of the next cell that needs no other thread: forward b d - c0 prev (k first
    // in CSR order), backward the rescaled input (k last)
    T part;
#pragma unroll
    for (int u = 0; u < kD; ++u) load(u, ring[u]);
    // the column's cell next to the slab, from the launch that took the slab before
    T prev = T(0);
    if (col_ok && !BWD && k0 > 0) prev = A.y[sys * vl + lay.at(i, j, k0 - 1)];
    if (col_ok && BWD && k1 < nz) prev = xout[(long long)nxy * depth];
    auto first = [&](const Cell &cl) {  // the input, scaled where the row is
      if (FACTOR) return cl.c[3];
      return PLAIN && !BWD ? cl.x : cl.x * cl.c[3];
    };
    part = first(ring[0]);
    if (!BWD) part = term(part, ring[0], 0, prev);
    const int steps = depth + TX + TY - 2;
    for (int s0 = 0; s0 < steps; s0 += kD) {
#pragma unroll
      for (int u = 0; u < kD; ++u) {
        if (s0 + u >= steps) break;  // the same for every compute warp
        const T c0 = ring[u].c[0], c1 = ring[u].c[1], c2 = ring[u].c[2];
        const int kk = k + step * u;
        const bool act = (unsigned)kk < (unsigned)depth;
        T vp = T(0), vq = T(0);
        if (act) {
          vp = W::peek(p_at + u * p_inc);
          vq = W::peek(q_at + u * q_inc);
        }
        if (W::sent(vp) || W::sent(vq)) {
          int it = 0;
          while (W::sent(vp) || W::sent(vq)) {
            vp = W::peek(p_at + u * p_inc);
            vq = W::peek(q_at + u * q_inc);
            if (++it > 32 * spin || ((it & 255) == 255 && *(volatile int *)&ctl[3])) {
              if (atomicExch(&ctl[3], 1) == 0) {
                if (fail) *fail = 1;
                atomicCAS(status, 0, FCG_ERR_TIMEOUT);
              }
              break;
            }
          }
        }
        T val;
        if (!BWD) {  // lower entries in CSR order: k, j, i
          val = term(part, ring[u], 1, vq);
          val = term(val, ring[u], 2, vp);
          if (FACTOR)
            val = T(1) / val;
          else if (PLAIN)
            val = val * ring[u].c[3];
        } else {  // upper entries in CSR order: i, j, k
          val = sub(part, c0, vp);
          val = sub(val, c1, vq);
          val = sub(val, c2, prev);
          if (PLAIN) val = val * ring[u].e[0];
        }
        // What the next step waits for comes before the barrier, stores to global memory after
        // it.  The loads: after the barrier in the forward sweep (153 -> 143 us at 128^3),
        // before it in the backward one, where after it costs 5 %.
        const Cell &next = ring[(u + 1) % kD];
        if (BWD) load(u + kD, ring[u]);
        part = first(next);
        sm[(u + 1) % kD][dj][di] = val;
        if (act) prev = val;
        if (!BWD) part = term(part, next, 0, prev);
        if (act && near_p) W::push(push_p + step * u * (int)sizeof(T), val);
        if (act && near_q) W::push(push_q + step * u * (int)sizeof(T), val);
        asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
        if (BWD) {
          if (act && col_ok) xout[(long long)nxy * kk] = val;
          if (act && far_out) W::st(zw + step * u * NT, val);
          if (act && rearm_y) yw[step * u * NT] = W::sentinel();
        } else {
          if (act) W::st(yw + step * u * NT, val);
          if (act && rearm_z) zw[step * u * NT] = W::sentinel();
          load(u + kD, ring[u]);
        }
      }
      k += step * kD;
      rec += step * kD * (P * NT);
      yw += step * kD * NT;
      zw += step * kD * NT;
      p_at += p_round;
      q_at += q_round;
      push_p += (uint32_t)(step * kD * (int)sizeof(T));
      push_q += (uint32_t)(step * kD * (int)sizeof(T));
    }
  }
  cluster.sync();  // no block leaves while a neighbour may store into its buffers
}

// f(cell row r, its position q in wavefront order, i, j, k) for the cells of the block, in
// wavefront order: a thread block takes kPackLevels levels of a tile at a time, so that its
// stores are whole lines and what it reads of the CSR row by row (consecutive cells in i
// stand on consecutive levels) is used up out of the first-level cache.  In row order every
// store was a sector of its own: five FP32 systems of 128^3 took 2.4 ms to pack, now 0.5.
constexpr int kPackLevels = 16;

template <class F>
__device__ __forceinline__ void for_cells(const Layout &lay, F &&f) {
  const int nch = (lay.nlev + kPackLevels - 1) / kPackLevels, items = lay.ntx * lay.nty * nch;
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int t = it / nch, L0 = (it - t * nch) * kPackLevels;
    const int i0 = t % lay.ntx * TX, j0 = t / lay.ntx * TY;
    for (int u = threadIdx.x; u < kPackLevels * NT; u += blockDim.x) {
      const int L = L0 + u / NT, c = u % NT, di = c % TX, dj = c / TX;
      const int i = i0 + di, j = j0 + dj, k = L - di - dj;
      if (i < lay.nx && j < lay.ny && k >= 0 && k < lay.nz)
        f(i + (long long)lay.nx * (j + (long long)lay.ny * k),
          ((long long)t * lay.nlev + L) * NT + c, i, j, k);
    }
  }
}

// Records of the factor of system blockIdx.y from the CSR values a (system s at s nnz).
template <class T, bool PLAIN>
__global__ void __launch_bounds__(kTPB)
    k_wave_pack_factor(int nx, int ny, int nz, long long nnz, const int *__restrict__ ioffset,
                       const int *__restrict__ diag, const int *__restrict__ tpos,
                       const T *__restrict__ a, int dilu, Arrays<T> A) {
  const Layout lay(nx, ny, nz);
  const int s = blockIdx.y;
  const T *as = a + s * nnz;
  T *fwd = A.fwd + s * lay.rec_len(), *bwd = A.bwd + s * lay.rec_len();
  for_cells(lay, [&](long long r, long long q, int i, int j, int k) {
    const long long at = q / NT * kPlanes * NT + q % NT;
    T *f = fwd + at, *b = bwd + at;
    int e = ioffset[r];
    const bool has[3] = {k > 0, j > 0, i > 0};
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      if (PLAIN) {
        f[p * NT] = has[p] ? as[e] : T(0);
        b[p * NT] = has[p] ? as[dilu ? tpos[e] : e] : T(0);
      } else {
        f[p * NT] = has[p] ? as[e] * (dilu ? as[tpos[e]] : as[e]) : T(0);
      }
      e += has[p];
    }
    f[3 * NT] = as[diag[r]];
  });
}

// Records of the sweeps of system blockIdx.y from the CSR values a (system s at s nnz) and
// the factor, which the factor sweep left in A.y; a pivot that is not finite is recorded.
template <class T, bool PLAIN>
__global__ void __launch_bounds__(kTPB)
    k_wave_pack(int nx, int ny, int nz, long long nnz, const int *__restrict__ ioffset,
                const int *__restrict__ diag, const T *__restrict__ a, T small, Arrays<T> A,
                int *status) {
  const Layout lay(nx, ny, nz);
  const int s = blockIdx.y;
  const T *as = a + s * nnz, *y = A.y + s * lay.vec_len();
  T *fwd = A.fwd + s * lay.rec_len(), *bwd = A.bwd + s * lay.rec_len();
  for_cells(lay, [&](long long r, long long q, int i, int j, int k) {
    const long long at = q / NT * kPlanes * NT + q % NT;
    const int lo = ioffset[r], up = diag[r] + 1;
    const bool l0 = k > 0, l1 = j > 0, l2 = i > 0;
    const bool u0 = i < nx - 1, u1 = j < ny - 1, u2 = k < nz - 1;
    T *f = fwd + at, *b = bwd + at;
    const T dd = y[q];
    auto coef = [&](bool has, int e) {
      if (!has) return T(0);
      return PLAIN ? as[e] : as[e] * dd;
    };
    f[0] = coef(l0, lo);
    f[NT] = coef(l1, lo + l0);
    f[2 * NT] = coef(l2, lo + l0 + l1);
    f[3 * NT] = dd;
    b[0] = coef(u0, up);
    b[NT] = coef(u1, up + u0);
    b[2 * NT] = coef(u2, up + u0 + u1);
    b[3 * NT] = (PLAIN ? T(1) : dd) / (dd + small);
    if (!isfinite(dd)) atomicCAS(status, 0, FCG_ERR_PIVOT);
  });
}

// Sentinels into the sweeps' vectors and the control words {forward claims, backward
// claims, -, error} cleared; before the first application of a solve.
template <class T>
__global__ void k_wave_arm(long long len, T *y, T *ze, int *ctl) {
  if (blockIdx.x == 0 && threadIdx.x < 4) ctl[threadIdx.x] = 0;
  FCG_GRID_STRIDE(i, len) {
    y[i] = Word<T>::sentinel();
    ze[i] = Word<T>::sentinel();
  }
}

// Is the factor formed in the PLAIN way?
template <class T, bool PLAIN>
constexpr bool kPlainFactor = PLAIN || sizeof(T) == 4;

// The arrays of ns systems on c's block, zeroed, and the kernels' shared-memory opt-in.
template <class T, bool PLAIN = false>
int allow_shared(fcg_context *c) {
  const int smem = (TX + TY) * kSlab * (int)sizeof(T);
  for (const void *f : {(const void *)k_wave_sweep<T, kForward, PLAIN>,
                        (const void *)k_wave_sweep<T, kBackward, PLAIN>,
                        (const void *)k_wave_sweep<T, kFactor, kPlainFactor<T, PLAIN>>})
    FCG_CUDA_TRY(c, cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  return FCG_OK;
}

template <class T>
size_t array_bytes(const Layout &lay, int ns) {
  return sizeof(T) * (size_t)ns * (size_t)(2 * lay.rec_len() + 2 * lay.vec_len());
}

// Does c's block take the wavefront form for ns systems?  The records hold a tile's whole
// wavefront, nz + 22 levels of 128 columns, which on a thin block is many times its cells:
// 12 times with two planes, 8 with two cells in i (2000 x 2000 x 2: 7.7 GB; level order,
// level_sweep.cuh, about 1.2).  Such a block goes over to level order where that is also the
// faster form, as its tiles, claimed row by row, number several times what the chip holds at
// once, and where the records would take more than 4 GB.  40 ICCG sweeps, ms, wavefront /
// level order: 512 x 512 x 2 (2048 tiles) 52 / 58; 724 x 724 x 2 (4186) 120 / 83; 2000 x 2000
// x 2 (31250) 1548 / 244; 2 x 2000 x 2000 (5.2 GB) 346 / 240.  Below both lines the wavefront
// form is up to twice as fast (128 x 128 x 2: 7.7 / 14.9; 2 x 1024 x 512: 53 / 83).
template <class T>
bool applies(const fcg_context *c, int ns) {
  if (!c->hex.ok) return false;
  const Layout lay(c->hex.nx, c->hex.ny, c->hex.nz);
  const bool thin = lay.len() > 4LL * c->n;
  return !thin || ((long long)lay.ntx * lay.nty * ns <= 16LL * c->num_sms &&
                   array_bytes<T>(lay, ns) <= (size_t)4 << 30);
}

// The column of a row that a block of another cluster waits for in the forward sweep, -1
// when there is none.
inline int awaited_column(const HexBlock &h, int row) {
  if (row < 0) return -1;
  const int i = row % h.nx, j = row / h.nx % h.ny;
  const bool p = i % (CX * TX) == CX * TX - 1 && i + 1 < h.nx;
  const bool q = j % (CY * TY) == CY * TY - 1 && j + 1 < h.ny;
  return p || q ? i + h.nx * j : -1;
}

template <class T>
int allocate(fcg_context *c, int ns, DBuf &buf, Arrays<T> &A) {
  const Layout lay(c->hex.nx, c->hex.ny, c->hex.nz);
  const long long g = Layout::guard(), rl = lay.rec_len(), vl = lay.vec_len();
  const size_t bytes = array_bytes<T>(lay, ns);
  FCG_CUDA_TRY(c, buf.ensure(bytes));
  FCG_CUDA_TRY(c, cudaMemsetAsync(buf.p, 0, bytes, c->stream));
  int rc = allow_shared<T>(c);
  if (!rc && sizeof(T) == 8) rc = allow_shared<T, sizeof(T) == 8>(c);
  if (rc) return rc;
  T *p = buf.as<T>();
  A.fwd = p + g;
  A.bwd = p + ns * rl + g;
  A.y = p + 2 * ns * rl + g;
  A.ze = p + ns * (2 * rl + vl) + g;
  return FCG_OK;
}

// What a launch needs besides the arrays: the solver's control words {forward claims,
// backward claims, -, error}, its status and stop flags (fail may be null) and the polls
// after which a wait gives up.
struct Control {
  int *ctl, *fail, *status;
  const int *done;
  int spin;
  // diagnostics (fcg_set_sweep_wait_test): the column i + nx j whose forward results never
  // reach the clusters that wait for them; -1: none
  int absent = -1;
  // the same without the solver's stop flag: the control word that stays zero
  Control unstopped() const { return Control{ctl, fail, status, ctl + 2, spin}; }
};

// One sweep, in launches of at most kSlab planes (each a whole sweep over its planes).
template <class T, bool PLAIN = false>
void launch(fcg_context *c, cudaStream_t st, int ns, int mode, const Arrays<T> &A, const T *in,
            T *out, const Control &w) {
  const HexBlock &h = c->hex;
  const int g = Layout(h.nx, h.ny, h.nz).clusters() * ns * CX * CY;
  const int slabs = (h.nz + kSlab - 1) / kSlab;
  for (int s = 0; s < slabs; ++s) {
    const int b = mode == kBackward ? slabs - 1 - s : s;
    const int k0 = (int)((long long)h.nz * b / slabs), k1 = (int)((long long)h.nz * (b + 1) / slabs);
    const size_t smem = (size_t)(TX + TY) * (k1 - k0) * sizeof(T);
    if (s > 0) cudaMemsetAsync(w.ctl, 0, 2 * sizeof(int), st);
    auto kernel = mode == kForward    ? k_wave_sweep<T, kForward, PLAIN>
                  : mode == kBackward ? k_wave_sweep<T, kBackward, PLAIN>
                                      : k_wave_sweep<T, kFactor, kPlainFactor<T, PLAIN>>;
    kernel<<<g, kThreads, smem, st>>>(h.nx, h.ny, h.nz, k0, k1, ns, A, in, out, w.ctl, w.fail,
                                      w.status, w.done, w.spin, w.absent);
  }
}

// The factor and the records of ns systems, and armed vectors: before the first sweep of
// a solve.  A pivot that breaks down is reported whether or not the first residual has
// already met the stop test.  128^3, FP64: about 0.2 ms; a factor that read the CSR at every step, with every
// hand-over through global memory, took 1.08 ms.
template <class T, bool PLAIN = false>
int start(fcg_context *c, int ns, long long nnz, const T *a, bool dilu, T small,
          const Arrays<T> &A, const Control &solver) {
  const Control w = solver.unstopped();
  const HexBlock &h = c->hex;
  const Layout lay(h.nx, h.ny, h.nz);
  const long long vl = ns * lay.vec_len(), g = Layout::guard();
  const int chunks = (lay.nlev + kPackLevels - 1) / kPackLevels;
  const int gv = grid_for(vl, c->num_sms);
  const dim3 gc(std::min(lay.ntx * lay.nty * chunks, c->num_sms * 8), ns);
  k_wave_pack_factor<T, kPlainFactor<T, PLAIN>><<<gc, kTPB, 0, c->stream>>>(h.nx, h.ny, h.nz, nnz, c->mv.ioffset,
                                                    c->mv.diag, c->tpos, a, dilu, A);
  k_wave_arm<T><<<gv, kTPB, 0, c->stream>>>(vl, A.y - g, A.ze - g, w.ctl);
  launch<T, PLAIN>(c, c->stream, ns, kFactor, A, nullptr, nullptr, w);
  k_wave_pack<T, PLAIN><<<gc, kTPB, 0, c->stream>>>(h.nx, h.ny, h.nz, nnz, c->mv.ioffset, c->mv.diag, a,
                                             small, A, w.status);
  k_wave_arm<T><<<gv, kTPB, 0, c->stream>>>(vl, A.y - g, A.ze - g, w.ctl);
  FCG_CHECK_LAUNCH(c, "wavefront factor and records");
  return FCG_OK;
}

}  // namespace wave
}  // namespace fcg
