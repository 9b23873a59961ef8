// The product of one message-passing layer of the learned preconditioner for the 16 cells
// of a warp, shared by every form of the layer kernel (learned.cu: the sliced gather form
// and the split form; learned_hex.cu: the plane-staged form for lexicographic hex meshes),
// so that all of them round identically.
//
// The 64 -> 32 product of the rows [h; m] runs as 4 k-steps x 4 n-blocks of
// mma.sync.m16n8k16 (BF16 operands, FP32 accumulation) on operands in registers (hpos),
// W_l's fragments from shared memory.  The epilogue adds the bias, applies the ReLU and
// the skip connection, h' = h + relu(W [h; m] + b).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace fcg {
namespace lp {

constexpr int kTileC = 32;                 // channels

__device__ __forceinline__ float bf(const __nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4], unsigned b0,
                                         unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Position of channel c in a stored activation row.  The rows keep their channels in the
// order of the mma.m16n8k16 fragments: the 16-byte quarter tg holds channels 8 i + 2 tg,
// + 1 for i = 0..3, which are the lane tg's columns of the A operand (two k-steps of 16
// channels) and of the result (four n-blocks).  A lane that holds a quarter of a row
// holds its fragments, and no value passes through shared memory on its way into or out
// of the product.
__host__ __device__ constexpr int hpos(int c) { return 8 * ((c >> 1) & 3) + 2 * (c >> 3) + (c & 1); }

// acc[0..7] = fma(v, 8 BF16 values packed in q, acc): one neighbour's term of m = Ahat h
// for eight channels.  The explicit fused multiply-add fixes the rounding for every
// kernel form.
__device__ __forceinline__ void fma8(float (&acc)[8], float v, const uint4 &q) {
  const __nv_bfloat162 *e = reinterpret_cast<const __nv_bfloat162 *>(&q);
  const float2 vv = make_float2(v, v);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    // packed FP32 FMA: each half is fma(v, h, acc), rounded to nearest
    const float2 r =
        __ffma2_rn(vv, __bfloat1622float2(e[c]), make_float2(acc[2 * c], acc[2 * c + 1]));
    acc[2 * c] = r.x;
    acc[2 * c + 1] = r.y;
  }
}

// The same with the neighbour's eight channels already in FP32.
__device__ __forceinline__ void fma8(float (&acc)[8], float v, const float (&h)[8]) {
  const float2 vv = make_float2(v, v);
#pragma unroll
  for (int c = 0; c < 8; c += 2) {
    const float2 r =
        __ffma2_rn(vv, make_float2(h[c], h[c + 1]), make_float2(acc[c], acc[c + 1]));
    acc[c] = r.x;
    acc[c + 1] = r.y;
  }
}

// Eight BF16 values to FP32, and back (of values that are BF16).
__device__ __forceinline__ void widen8(float (&h)[8], const uint4 &q) {
  const __nv_bfloat162 *e = reinterpret_cast<const __nv_bfloat162 *>(&q);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float2 f = __bfloat1622float2(e[c]);
    h[2 * c] = f.x;
    h[2 * c + 1] = f.y;
  }
}
__device__ __forceinline__ uint4 narrow8(const float (&h)[8]) {
  unsigned r[4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
    r[c] = __byte_perm(__float_as_uint(h[2 * c]), __float_as_uint(h[2 * c + 1]), 0x7632);
  return make_uint4(r[0], r[1], r[2], r[3]);
}

// The network's output before its scaling, w_out . h + b_out, over one BF16 row of
// kTileC channels held in v, in channel order (w = [w_out, b_out]).
__device__ __forceinline__ float out_dot_vals(const uint4 (&v)[4], const float *w) {
  float acc = w[kTileC];
#pragma unroll
  for (int c = 0; c < kTileC; ++c)
    acc += w[c] * bf(reinterpret_cast<const __nv_bfloat16 *>(&v[hpos(c) >> 3])[hpos(c) & 7]);
  return acc;
}

// out_dot_vals of a row in shared memory (16-byte aligned).
__device__ __forceinline__ float out_dot_row(const __nv_bfloat16 *row, const float *w) {
  uint4 v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = reinterpret_cast<const uint4 *>(row)[q];
  return out_dot_vals(v, w);
}

// W_l as B fragments in shared memory (4 KB): entry (2 kb + p) 32 + lane holds the lane's
// fragments of k-step kb for the n-blocks 2 p and 2 p + 1.
constexpr int kFragWords = 8 * 32;
__device__ __forceinline__ void load_frags(uint4 *wf, const __nv_bfloat16 *__restrict__ wl) {
  for (int t = threadIdx.x; t < kFragWords; t += blockDim.x) {
    const int kb = t >> 6, p = (t >> 5) & 1, g = (t >> 2) & 7, tg = t & 3;
    unsigned v[4];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const __nv_bfloat16 *w = wl + (8 * (2 * p + s) + g) * 2 * kTileC + 16 * kb + 2 * tg;
      v[2 * s] = *reinterpret_cast<const unsigned *>(w);
      v[2 * s + 1] = *reinterpret_cast<const unsigned *>(w + 8);
    }
    wf[t] = make_uint4(v[0], v[1], v[2], v[3]);
  }
}
// The lane's biases: channels 8 nt + 2 tg, + 1.
__device__ __forceinline__ void load_bias(float (&bias)[8], const float *b, int lane) {
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    bias[2 * nt] = b[nt * 8 + 2 * (lane & 3)];
    bias[2 * nt + 1] = b[nt * 8 + 2 * (lane & 3) + 1];
  }
}

// Eight FP32 sums to BF16, packed.
__device__ __forceinline__ uint4 round8(const float (&acc)[8]) {
  uint4 q;
  __nv_bfloat162 *e = reinterpret_cast<__nv_bfloat162 *>(&q);
#pragma unroll
  for (int c = 0; c < 4; ++c) e[c] = __floats2bfloat162_rn(acc[2 * c], acc[2 * c + 1]);
  return q;
}

// The product and epilogue of 16 rows, h' = h + relu(W_l [h; m] + b): lane 4 g + tg holds
// the quarters tg of rows g and g + 8 (own: h, m) and receives theirs of h'.
// zout(row, channel, z0, z1) receives the pre-activations of channels channel, + 1
// (training); pass a no-op otherwise.
template <class ZOut>
__device__ __forceinline__ void dense(const uint4 (&own)[2], const uint4 (&m)[2], const uint4 *wf,
                                      const float (&bias)[8], int lane, uint4 (&out)[2],
                                      ZOut zout) {
  const int g = lane >> 2, tg = lane & 3;
  float d[4][4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int q = 0; q < 4; ++q) d[nt][q] = 0.f;
#pragma unroll
  for (int kb = 0; kb < 4; ++kb) {
    const uint4 &x = kb < 2 ? own[0] : m[0], &y = kb < 2 ? own[1] : m[1];
    const unsigned a[4] = {kb & 1 ? x.z : x.x, kb & 1 ? y.z : y.x, kb & 1 ? x.w : x.y,
                           kb & 1 ? y.w : y.y};
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const uint4 b = wf[(2 * kb + p) * 32 + lane];
      mma_bf16(d[2 * p], a, b.x, b.y);
      mma_bf16(d[2 * p + 1], a, b.z, b.w);
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const __nv_bfloat162 *hold = reinterpret_cast<const __nv_bfloat162 *>(&own[r]);
    __nv_bfloat162 *o = reinterpret_cast<__nv_bfloat162 *>(&out[r]);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const float2 z = __fadd2_rn(make_float2(d[nt][2 * r], d[nt][2 * r + 1]),
                                  make_float2(bias[2 * nt], bias[2 * nt + 1]));
      o[nt] = __float22bfloat162_rn(__fadd2_rn(
          __bfloat1622float2(hold[nt]), make_float2(fmaxf(z.x, 0.f), fmaxf(z.y, 0.f))));
      zout(g + 8 * r, nt * 8 + 2 * tg, z.x, z.y);
    }
  }
}

struct NoZ {
  __device__ __forceinline__ void operator()(int, int, float, float) const {}
};

}  // namespace lp
}  // namespace fcg
