// Cell-centred gradients and boundary values: grad_gauss (grad_gauss.f90),
// grad_gauss_corrected (grad_gauss_corrected.f90), grad_lsq (grad_lsq.f90) and
// bpres (bpres.f90).
//
// Gauss: one thread per inner face computes the interpolated face value times the
// area vector (gradco :128-190) into a face array; one thread per cell then adds its
// inner faces in face order (+ as owner, - as neighbour), its boundary faces in the
// reference's boundary-loop order (gradbc :194-211) and scales by 1/vol, straight into the
// caller's array.  LSQ: one
// thread per cell gathers the same per-face terms the reference scatters.  Compiled
// with --fmad=false, so results are bit-identical to the Fortran loops.
#include "fcg_internal.h"
#include "launch.h"

using namespace fcg;

namespace {

// The bound mesh's constants of the Gauss gradient: 1/vol per cell, and `odd`, set where a
// face's interpolation factors or offset are not finite.
struct GaussConst {
  const double *volr;
  const int *odd;
};

struct FaceOffset {
  double fxn, fxp, dx, dy, dz;
};

// Face f between cells p and q with factor fxn: the offset of the face centre from the
// interpolation point on PN.
__device__ __forceinline__ FaceOffset face_offset(const MeshView &m, long long f, int p, int q,
                                                  double fxn) {
  const double fxp = 1.0 - fxn;
  const double xi = m.xc[p] * fxp + m.xc[q] * fxn;
  const double yi = m.yc[p] * fxp + m.yc[q] * fxn;
  const double zi = m.zc[p] * fxp + m.zc[q] * fxn;
  return {fxn, fxp, m.xf[f] - xi, m.yf[f] - yi, m.zf[f] - zi};
}

__global__ void k_gauss_const(MeshView m, double *__restrict__ volr, int *__restrict__ odd) {
  FCG_GRID_STRIDE(c, m.n) volr[c] = 1.0 / m.vol[c];
  FCG_GRID_STRIDE(f, m.nin) {
    const FaceOffset o = face_offset(m, f, m.owner[f], m.neighbour[f], m.facint[f]);
    if (!(isfinite(o.fxn) && isfinite(o.fxp) && isfinite(o.dx) && isfinite(o.dy) &&
          isfinite(o.dz)))
      *odd = 1;
  }
}

// gradco: face value with the old gradient (zero without gold) interpolated to the point
// on PN.
__device__ __forceinline__ double face_value(const FaceOffset &o, int p, int q,
                                             const double *__restrict__ fi,
                                             const double *__restrict__ gold) {
  auto old = [&](int c, int k) { return gold ? gold[3LL * c + k] : 0.0; };
  const double dfxi = old(p, 0) * o.fxp + old(q, 0) * o.fxn;
  const double dfyi = old(p, 1) * o.fxp + old(q, 1) * o.fxn;
  const double dfzi = old(p, 2) * o.fxp + old(q, 2) * o.fxn;
  return fi[p] * o.fxp + fi[q] * o.fxn + dfxi * o.dx + dfyi * o.dy + dfzi * o.dz;
}

// Bound by the FP64 pipe (629 G instructions/s): 34 of them a face with an old gradient,
// 7 without (FIRST, the first pass).  With a zero gradient and finite factors the
// correction terms are products with zero: adding them changes no bit of the face's
// contribution (a zero's sign is lost in the cell's sum, which starts from +0), so the
// first pass leaves them out and reads neither the cell centres nor the face centres.
// Factors that are not finite would make those products NaN; such a mesh (odd) takes
// the whole expression.  6.2 M faces (128^3): 94 us, with the zero terms 432.
template <bool FIRST>
__global__ void __launch_bounds__(kTPB)
    k_gauss_faces(MeshView m, GaussConst k, const double *__restrict__ fi,
                  const double *__restrict__ gold, double *__restrict__ dfe) {
  const bool plain = FIRST && __ldg(k.odd) == 0;
  FCG_GRID_STRIDE(f, m.nin) {
    const int p = m.owner[f], q = m.neighbour[f];
    const double fxn = m.facint[f];
    double fie;
    if (plain)
      fie = fi[p] * (1.0 - fxn) + fi[q] * fxn;
    else
      fie = face_value(face_offset(m, f, p, q, fxn), p, q, fi, FIRST ? nullptr : gold);
    dfe[f] = fie * m.arx[f];
    dfe[m.nin + f] = fie * m.ary[f];
    dfe[2LL * m.nin + f] = fie * m.arz[f];
  }
}

// The same on the O-C pairs (grad_gauss.f90:60-67): face ijlFace(i), factor foc(i).
__global__ void k_gauss_oc(MeshView m, const double *__restrict__ fi,
                           const double *__restrict__ gold, double *__restrict__ dfo) {
  FCG_GRID_STRIDE(i, m.noc) {
    const int p = m.oc_l[i], q = m.oc_r[i], f = m.oc_fl[i];
    const double fie = face_value(face_offset(m, f, p, q, m.oc_foc[i]), p, q, fi, gold);
    dfo[i] = fie * m.arx[f];
    dfo[m.noc + i] = fie * m.ary[f];
    dfo[2LL * m.noc + i] = fie * m.arz[f];
  }
}

constexpr int kBatch = 3;

// Bound by the FP64 pipe: 21 instructions a cell (1/vol is the mesh's, and the sign of a
// neighbour's term an integer flip).  128^3: 106 us; with a quotient and two signed sums a
// face 208, with negations in FP64 189.  Batches of 2, 3 and 6 faces differ by 2 %.
__global__ void __launch_bounds__(kTPB)
    k_gauss_cells(MeshView m, GaussConst k, const double *__restrict__ fi,
                  const double *__restrict__ dfe, const double *__restrict__ dfo,
                  double *__restrict__ g) {
  FCG_GRID_STRIDE(c, m.n) {
    double gx = 0.0, gy = 0.0, gz = 0.0;
    // the loads of kBatch faces are issued together; added in face order, + as owner, - as
    // neighbour (x - e is x + (-e) to the bit)
    const int e1 = m.cf_ptr[c + 1];
    for (int e = m.cf_ptr[c]; e < e1; e += kBatch) {
      int ent[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) ent[u] = e + u < e1 ? m.cf_ent[e + u] : 0;
      double t[kBatch][3];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const long long f = (ent[u] > 0 ? ent[u] : -ent[u]) - 1;
#pragma unroll
        for (int k = 0; k < 3; ++k) t[u][k] = ent[u] ? dfe[(long long)k * m.nin + f] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        if (!ent[u]) break;
        const bool own = ent[u] > 0;
        gx = gx + signed_term(own, t[u][0]);
        gy = gy + signed_term(own, t[u][1]);
        gz = gz + signed_term(own, t[u][2]);
      }
    }
    if (m.noc)  // the O-C pairs after the inner faces, + on the left cell, - on the right
      for (int e = m.oc_cptr[c]; e < m.oc_cptr[c + 1]; ++e) {
        const int v = m.oc_vix[e];
        const long long i = v < m.noc ? v : v - m.noc;
        double ex = dfo[i], ey = dfo[m.noc + i], ez = dfo[2LL * m.noc + i];
        if (v < m.noc) {
          gx = gx + ex;
          gy = gy + ey;
          gz = gz + ez;
        } else {
          gx = gx - ex;
          gy = gy - ey;
          gz = gz - ez;
        }
      }
    for (int e = m.cb_ptr[c]; e < m.cb_ptr[c + 1]; ++e) {
      int f = m.cb_face[e];
      double fb = fi[m.cb_slot[e]];
      gx = gx + fb * m.arx[f];
      gy = gy + fb * m.ary[f];
      gz = gz + fb * m.arz[f];
    }
    const double volr = k.volr[c];
    g[3 * c] = gx * volr;
    g[3 * c + 1] = gy * volr;
    g[3 * c + 2] = gz * volr;
  }
}

// grad_lsq stage 1: D = sum d d^T over inner faces (face order) and boundary faces
// (face order), then the scaled cofactors (:134-165).
__global__ void k_lsq_matrix(MeshView m, double *__restrict__ dmat) {
  FCG_GRID_STRIDE(c, m.n) {
    double d11 = 0.0, d12 = 0.0, d13 = 0.0, d22 = 0.0, d23 = 0.0, d33 = 0.0;
    for (int e = m.cf_ptr[c]; e < m.cf_ptr[c + 1]; ++e) {
      int ent = m.cf_ent[e];
      int f = (ent > 0 ? ent : -ent) - 1;
      int p = m.owner[f], q = m.neighbour[f];
      double Dx = m.xc[q] - m.xc[p], Dy = m.yc[q] - m.yc[p], Dz = m.zc[q] - m.zc[p];
      d11 = d11 + Dx * Dx;
      d22 = d22 + Dy * Dy;
      d33 = d33 + Dz * Dz;
      d12 = d12 + Dx * Dy;
      d13 = d13 + Dx * Dz;
      d23 = d23 + Dy * Dz;
    }
    if (m.noc)  // the O-C pairs (:85-108)
      for (int e = m.oc_cptr[c]; e < m.oc_cptr[c + 1]; ++e) {
        const int v = m.oc_vix[e], i = v < m.noc ? v : v - m.noc;
        const int p = m.oc_l[i], q = m.oc_r[i];
        double Dx = m.xc[q] - m.xc[p], Dy = m.yc[q] - m.yc[p], Dz = m.zc[q] - m.zc[p];
        d11 = d11 + Dx * Dx;
        d22 = d22 + Dy * Dy;
        d33 = d33 + Dz * Dz;
        d12 = d12 + Dx * Dy;
        d13 = d13 + Dx * Dz;
        d23 = d23 + Dy * Dz;
      }
    for (int e = m.cbf_ptr[c]; e < m.cbf_ptr[c + 1]; ++e) {
      int f = m.cbf_face[e];
      double Dx = m.xf[f] - m.xc[c], Dy = m.yf[f] - m.yc[c], Dz = m.zf[f] - m.zc[c];
      d11 = d11 + Dx * Dx;
      d22 = d22 + Dy * Dy;
      d33 = d33 + Dz * Dz;
      d12 = d12 + Dx * Dy;
      d13 = d13 + Dx * Dz;
      d23 = d23 + Dy * Dz;
    }
    double d21 = d12, d31 = d13, d32 = d23;
    double tmp = 1.0 / (d11 * d22 * d33 - d11 * d23 * d32 - d12 * d21 * d33 + d12 * d23 * d31 +
                        d13 * d21 * d32 - d13 * d22 * d31);
    double *D = dmat + 9 * c;
    D[0] = (d22 * d33 - d23 * d32) * tmp;
    D[1] = (d21 * d33 - d23 * d31) * tmp;
    D[2] = (d21 * d32 - d22 * d31) * tmp;
    D[3] = (d11 * d33 - d13 * d31) * tmp;
    D[4] = (d12 * d33 - d13 * d32) * tmp;
    D[5] = (d11 * d32 - d12 * d31) * tmp;
    D[6] = (d12 * d23 - d13 * d22) * tmp;
    D[7] = (d11 * d23 - d13 * d21) * tmp;
    D[8] = (d11 * d22 - d12 * d21) * tmp;
  }
}

// grad_lsq stage 2 (:168-306).
__global__ void k_lsq_cells(MeshView m, const double *__restrict__ fi,
                            const double *__restrict__ dmat, double *__restrict__ g) {
  FCG_GRID_STRIDE(c, m.n) {
    double b1 = 0.0, b2 = 0.0, b3 = 0.0;
    for (int e = m.cf_ptr[c]; e < m.cf_ptr[c + 1]; ++e) {
      int ent = m.cf_ent[e];
      int f = (ent > 0 ? ent : -ent) - 1;
      int p = m.owner[f], q = m.neighbour[f];
      double df = fi[q] - fi[p];
      b1 = b1 + (m.xc[q] - m.xc[p]) * df;
      b2 = b2 + (m.yc[q] - m.yc[p]) * df;
      b3 = b3 + (m.zc[q] - m.zc[p]) * df;
    }
    if (m.noc)  // the O-C pairs (:198-214)
      for (int e = m.oc_cptr[c]; e < m.oc_cptr[c + 1]; ++e) {
        const int v = m.oc_vix[e], i = v < m.noc ? v : v - m.noc;
        const int p = m.oc_l[i], q = m.oc_r[i];
        double df = fi[q] - fi[p];
        b1 = b1 + (m.xc[q] - m.xc[p]) * df;
        b2 = b2 + (m.yc[q] - m.yc[p]) * df;
        b3 = b3 + (m.zc[q] - m.zc[p]) * df;
      }
    for (int e = m.cb_ptr[c]; e < m.cb_ptr[c + 1]; ++e) {
      int f = m.cb_face[e];
      double df = fi[m.cb_slot[e]] - fi[c];
      b1 = b1 + df * (m.xf[f] - m.xc[c]);
      b2 = b2 + df * (m.yf[f] - m.yc[c]);
      b3 = b3 + df * (m.zf[f] - m.zc[c]);
    }
    const double *D = dmat + 9 * c;
    g[3 * c] = b1 * D[0] - b2 * D[1] + b3 * D[2];
    g[3 * c + 1] = b1 * D[3] - b2 * D[4] - b3 * D[5];
    g[3 * c + 2] = b1 * D[6] - b2 * D[7] + b3 * D[8];
  }
}

// bpres: one thread per boundary face listed by type; each writes its own slot.
__global__ void k_bpres(MeshView m, long long nbent, double *__restrict__ p,
                        const double *__restrict__ dP, int istage) {
  FCG_GRID_STRIDE(e, nbent) {
    int f = m.cb_face[e], c = m.owner[f], slot = m.cb_slot[e], t = m.cb_type[e];
    if (istage == 1) {
      p[slot] = p[c];  // :37-96
    } else if (t == B_WALL || t == B_PRESSOUT) {  // :102-132
      double xpb = m.xf[f] - m.xc[c], ypb = m.yf[f] - m.yc[c], zpb = m.zf[f] - m.zc[c];
      p[slot] = p[c] + dP[3 * c] * xpb + dP[3 * c + 1] * ypb + dP[3 * c + 2] * zpb;
    }
  }
}

// bpres on the O-C slots (:89-95, :134-148): slot s0 + i takes the value of the owner of
// face iOCFacesStart + i; from stage 2 on, extrapolated over the distance from the
// centre of face i, as :140-142 write it.
__global__ void k_bpres_oc(MeshView m, long long s0, double *__restrict__ p,
                           const double *__restrict__ dP, int istage) {
  FCG_GRID_STRIDE(i, m.noc) {
    const int c = m.owner[m.oc_start + i];
    if (istage == 1) {
      p[s0 + i] = p[c];
    } else {
      double xpb = m.xf[i] - m.xc[c], ypb = m.yf[i] - m.yc[c], zpb = m.zf[i] - m.zc[c];
      p[s0 + i] = p[c] + dP[3 * c] * xpb + dP[3 * c + 1] * ypb + dP[3 * c + 2] * zpb;
    }
  }
}

int ensure_gauss_const(fcg_context *c, GaussConst *k) {
  const size_t nv = sizeof(double) * (size_t)c->n;
  if (!c->gconst_ready) {
    FCG_CUDA_TRY(c, c->gconst.ensure(nv + sizeof(int)));
    double *volr = c->gconst.as<double>();
    FCG_CUDA_TRY(c, cudaMemsetAsync(volr + c->n, 0, sizeof(int), c->stream));
    const int g = grid_for(std::max(c->mv.n, c->mv.nin), c->num_sms);
    k_gauss_const<<<g, kTPB, 0, c->stream>>>(c->mv, volr, (int *)(volr + c->n));
    FCG_CHECK_LAUNCH(c, "k_gauss_const");
    c->gconst_ready = true;
  }
  *k = {c->gconst.as<double>(), (const int *)(c->gconst.as<double>() + c->n)};
  return FCG_OK;
}

// Do the byte ranges [a, a + na) and [b, b + nb) share a byte?
bool overlap(const void *a, size_t na, const void *b, size_t nb) {
  const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
  return x < y + nb && y < x + na;
}

int ensure_lsq_matrix(fcg_context *c) {
  if (c->dmat_ready) return FCG_OK;
  FCG_CUDA_TRY(c, c->dmat.ensure(sizeof(double) * 9 * (size_t)c->n));
  k_lsq_matrix<<<grid_for(c->n, c->num_sms), kTPB, 0, c->stream>>>(c->mv, c->dmat.as<double>());
  FCG_CHECK_LAUNCH(c, "k_lsq_matrix");
  c->dmat_ready = true;
  return FCG_OK;
}

}  // namespace

extern "C" int fcg_grad_lsq_matrix(fcg_context *c, double *dmat) {
  if (!c) return FCG_ERR_ARG;
  if (!c->bound) return set_error(c, FCG_ERR_STATE, "fcg_grad_lsq_matrix before fcg_bind_mesh");
  FCG_CUDA_TRY(c, cudaSetDevice(c->device));
  c->dmat_ready = false;
  int rc = ensure_lsq_matrix(c);
  if (rc) return rc;
  if (dmat) {
    FCG_CUDA_TRY(c, cudaMemcpyAsync(dmat, c->dmat.p, sizeof(double) * 9 * (size_t)c->n,
                                    cudaMemcpyDefault, c->stream));
    FCG_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  }
  return FCG_OK;
}

extern "C" int fcg_grad(fcg_context *c, const double *phi, double *dPhidxi, int method,
                        int nigrad) {
  if (!c) return FCG_ERR_ARG;
  if (!c->bound) return set_error(c, FCG_ERR_STATE, "fcg_grad before fcg_bind_mesh");
  if (method != FCG_GRAD_GAUSS && method != FCG_GRAD_GAUSS_CORRECTED && method != FCG_GRAD_LSQ)
    return set_error(c, FCG_ERR_ARG, "unknown gradient method");
  if (method == FCG_GRAD_GAUSS && nigrad < 1)
    return set_error(c, FCG_ERR_ARG, "nigrad must be >= 1");
  FCG_CUDA_TRY(c, cudaSetDevice(c->device));
  const size_t n3 = sizeof(double) * 3 * (size_t)c->n;
  void *dphi, *dg;
  bool hphi, hg;
  int rc;
  if ((rc = stage_in(c, phi, sizeof(double) * c->ntot, 0, true, &dphi, &hphi))) return rc;
  if ((rc = stage_in(c, dPhidxi, n3, 1, method == FCG_GRAD_GAUSS_CORRECTED, &dg, &hg))) return rc;
  const MeshView &m = c->mv;
  // several waves of blocks: a block's start hides another's last loads (8 an SM: 256 us a
  // pass at 128^3, 32: 232)
  const int gf = grid_for(m.nin, c->num_sms, 32), gc = grid_for(m.n, c->num_sms, 32);
  if (method == FCG_GRAD_LSQ) {
    if ((rc = ensure_lsq_matrix(c))) return rc;
    k_lsq_cells<<<gc, kTPB, 0, c->stream>>>(m, (const double *)dphi, c->dmat.as<double>(),
                                            (double *)dg);
    FCG_CHECK_LAUNCH(c, "k_lsq_cells");
  } else {
    // scratch: dfe[3*nin] | O-C terms [3*noc] | gradient [3n], if the result's array
    // shares memory with phi.  A pass reads the old gradient in its face kernels only, so
    // its cell kernel writes the new one over it (:116-120).
    const bool apart = !overlap(dphi, sizeof(double) * c->ntot, dg, n3);
    const size_t nin3 = 3 * (size_t)(m.nin > 0 ? m.nin : 1), noc3 = 3 * (size_t)m.noc;
    FCG_CUDA_TRY(c, c->scratch.ensure(sizeof(double) * (nin3 + noc3) + (apart ? 0 : n3)));
    GaussConst k;
    if ((rc = ensure_gauss_const(c, &k))) return rc;
    double *dfe = c->scratch.as<double>(), *dfo = dfe + nin3;
    double *g = apart ? (double *)dg : dfo + noc3;
    const int passes = method == FCG_GRAD_GAUSS_CORRECTED ? 1 : nigrad;
    // old gradient: incoming (grad_gauss_corrected.f90:38-40) or zero (grad_gauss.f90:38-40)
    const double *gold = method == FCG_GRAD_GAUSS_CORRECTED ? (const double *)dg : nullptr;
    for (int lc = 1; lc <= passes; ++lc) {
      if (m.nin > 0) {
        auto faces = gold ? k_gauss_faces<false> : k_gauss_faces<true>;
        faces<<<gf, kTPB, 0, c->stream>>>(m, k, (const double *)dphi, gold, dfe);
        FCG_CHECK_LAUNCH(c, "k_gauss_faces");
      }
      if (m.noc > 0) {
        k_gauss_oc<<<grid_for(m.noc, c->num_sms), kTPB, 0, c->stream>>>(m, (const double *)dphi,
                                                                         gold, dfo);
        FCG_CHECK_LAUNCH(c, "k_gauss_oc");
      }
      k_gauss_cells<<<gc, kTPB, 0, c->stream>>>(m, k, (const double *)dphi, dfe, dfo, g);
      FCG_CHECK_LAUNCH(c, "k_gauss_cells");
      gold = g;
    }
    if (!apart) FCG_CUDA_TRY(c, cudaMemcpyAsync(dg, g, n3, cudaMemcpyDeviceToDevice, c->stream));
  }
  if ((rc = stage_out(c, dPhidxi, dg, n3, hg))) return rc;
  if (hg) FCG_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  return FCG_OK;
}

extern "C" int fcg_bpres(fcg_context *c, double *p, const double *dPdxi, int istage) {
  if (!c) return FCG_ERR_ARG;
  if (!c->bound) return set_error(c, FCG_ERR_STATE, "fcg_bpres before fcg_bind_mesh");
  if (istage < 1) return set_error(c, FCG_ERR_ARG, "istage must be >= 1");
  FCG_CUDA_TRY(c, cudaSetDevice(c->device));
  void *dp, *dg = nullptr;
  bool hp, hg = false;
  int rc;
  if ((rc = stage_in(c, p, sizeof(double) * c->ntot, 0, true, &dp, &hp))) return rc;
  if (istage >= 2) {
    if ((rc = stage_in(c, dPdxi, sizeof(double) * 3 * (size_t)c->n, 1, true, &dg, &hg))) return rc;
  }
  long long nbent = 0;
  for (int t = 0; t < B_NTYPES; ++t) nbent += c->cnt[t];
  if (nbent > 0) {
    k_bpres<<<grid_for(nbent, c->num_sms), kTPB, 0, c->stream>>>(c->mv, nbent, (double *)dp,
                                                                   (const double *)dg, istage);
    FCG_CHECK_LAUNCH(c, "k_bpres");
  }
  if (c->mv.noc > 0) {  // the O-C slots follow the typed ones (iOCStart, :603)
    k_bpres_oc<<<grid_for(c->mv.noc, c->num_sms), kTPB, 0, c->stream>>>(
        c->mv, (long long)c->n + nbent, (double *)dp, (const double *)dg, istage);
    FCG_CHECK_LAUNCH(c, "k_bpres_oc");
  }
  if ((rc = stage_out(c, p, dp, sizeof(double) * c->ntot, hp))) return rc;
  if (hp) FCG_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  return FCG_OK;
}
