// The level order of a bound mesh's triangular sweeps (LevelOrder in fcg_internal.h), built
// from the CSR pattern and the padded level lists at the first solve that sweeps in it:
// position of every row, and per chunk of 32 positions the positions its rows read, column
// by column, with the CSR positions of their coefficients.
#include "fcg_internal.h"
#include "launch.h"

using namespace fcg;

namespace {

__global__ void k_positions(int len, const int *__restrict__ row, int *__restrict__ pos) {
  FCG_GRID_STRIDE(p, len) if (row[p] >= 0) pos[row[p]] = (int)p;
}

__device__ __forceinline__ void side_range(const int *ioffset, const int *diag, int upper, int r,
                                           int &b, int &e) {
  b = upper ? diag[r] + 1 : ioffset[r];
  e = upper ? ioffset[r + 1] : diag[r];
}

// entries of the widest row of every chunk
__global__ void k_widths(int len, const int *__restrict__ row, const int *__restrict__ ioffset,
                         const int *__restrict__ diag, int upper, int *__restrict__ width) {
  FCG_GRID_STRIDE(p, len) {  // len is a multiple of 32: whole warps
    int b = 0, e = 0;
    if (row[p] >= 0) side_range(ioffset, diag, upper, row[p], b, e);
    const int w = __reduce_max_sync(0xffffffffu, e - b);
    if ((p & 31) == 0) width[p >> 5] = w;
  }
}

__global__ void k_entries(int len, const int *__restrict__ row, const int *__restrict__ ioffset,
                          const int *__restrict__ ja, const int *__restrict__ diag, int upper,
                          const int *__restrict__ ptr, const int *__restrict__ pos,
                          int *__restrict__ dep, int *__restrict__ src) {
  FCG_GRID_STRIDE(p, len) {
    int b = 0, e = 0;
    if (row[p] >= 0) side_range(ioffset, diag, upper, row[p], b, e);
    for (int t = ptr[p >> 5]; t < ptr[(p >> 5) + 1]; ++t, ++b) {
      const long long q = 32LL * t + (p & 31);
      dep[q] = b < e ? pos[ja[b]] : -1;
      src[q] = b < e ? b : -1;
    }
  }
}

__global__ void k_other_positions(int len, const int *__restrict__ row,
                                  const int *__restrict__ pos, int *__restrict__ xpos) {
  FCG_GRID_STRIDE(p, len) xpos[p] = row[p] >= 0 ? pos[row[p]] : 0;
}

int build_side(fcg_context *c, const Level &lv, bool upper, LevelSide &s, int **pos,
               const int *lower_pos) {
  const MeshView &m = c->mv;
  const int len = lv.pad_len, chunks = len / 32, g = grid_for(len, c->num_sms);
  DBuf tmp, width, own;  // own: the side's arrays, kept with the bound mesh
  auto drop = [&] {
    tmp.release();
    width.release();
    own.release();
  };
  auto fail = [&](cudaError_t e, const char *what) {
    drop();
    return cuda_fail(c, e, what);
  };
  cudaError_t e;
  const size_t head = (size_t)chunks + 1 + (size_t)len;  // ptr, xpos
  if ((e = width.ensure(sizeof(int) * ((size_t)chunks + (size_t)chunks + 1)))) return fail(e, "widths");
  int *w = width.as<int>(), *wp = w + chunks;
  k_widths<<<g, kTPB, 0, c->stream>>>(len, lv.pad, m.ioffset, m.diag, upper, w);
  int rc = scan_ints(c, w, wp, chunks, tmp);
  if (rc) {
    drop();  // the scan has described its error
    return rc;
  }
  int total = 0;
  if ((e = cudaMemcpyAsync(&total, wp + chunks, sizeof(int), cudaMemcpyDeviceToHost, c->stream)) ||
      (e = cudaStreamSynchronize(c->stream)))
    return fail(e, "level widths");
  if ((e = own.ensure(sizeof(int) * (head + 64 * (size_t)total + (size_t)c->n))))
    return fail(e, "level order");
  int *ptr = own.as<int>(), *xpos = ptr + chunks + 1, *dep = xpos + len;
  int *src = dep + 32 * (size_t)total;
  *pos = src + 32 * (size_t)total;
  if ((e = cudaMemcpyAsync(ptr, wp, sizeof(int) * ((size_t)chunks + 1), cudaMemcpyDeviceToDevice,
                           c->stream)))
    return fail(e, "level order");
  k_positions<<<g, kTPB, 0, c->stream>>>(len, lv.pad, *pos);
  k_entries<<<g, kTPB, 0, c->stream>>>(len, lv.pad, m.ioffset, m.ja, m.diag, upper, ptr, *pos, dep,
                                       src);
  if (lower_pos) k_other_positions<<<g, kTPB, 0, c->stream>>>(len, lv.pad, lower_pos, xpos);
  if ((e = cudaGetLastError()) || (e = cudaStreamSynchronize(c->stream)))
    return fail(e, "level order");
  tmp.release();
  width.release();
  c->bound_allocs.push_back(own);
  s = LevelSide{chunks, total, lv.pad, ptr, dep, src, xpos};
  return FCG_OK;
}

}  // namespace

int fcg::level_order(fcg_context *c) {
  if (c->order.ready) return FCG_OK;
  int *pf = nullptr, *pb = nullptr;
  int rc = build_side(c, c->lf, false, c->order.lo, &pf, nullptr);
  if (!rc) rc = build_side(c, c->lb, true, c->order.up, &pb, pf);
  c->order.ready = rc == FCG_OK;
  return rc;
}
