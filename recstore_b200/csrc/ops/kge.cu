// Knowledge-graph embedding scoring with chunked shared negatives and the log-sigmoid loss, forward
// and backward, for six score functions: TransE (L2 and L1), DistMult, ComplEx, SimplE, RotatE.
//
// Math of the reference (src/kg/kg/dgl-ke/python/dglke/models/pytorch/score_fun.py:26-108 TransE,
// 222-286 DistMult, 288-368 ComplEx, 440-538 RotatE, 540-641 SimplE; loss.py:69-99;
// general_models.py:568-631).  A batch of `bs` positives is cut into chunks of `cs`; every chunk
// shares `ns` negative entities; loss = ( mean(-logsigmoid(pos)) + mean(-logsigmoid(-neg)) ) / 2.
// With x the entity that is kept (h when tails are corrupted, t when heads are) and y the other one,
// every model is  score = f( a(x, r), e )  with e = y for the positive and e = a negative entity:
//   TransE_l2  a = h + r | t - r                     score = gamma - ||a - e||_2
//   DistMult   a = x * r                             score = a . e
//   ComplEx    a = x (*) r | x (*) conj(r)           score = a . e      (entities are [re | im] halves)
//   SimplE     a = [x_j * r_inv | x_i * r] / 2 (tails) or [x_j * r | x_i * r_inv] / 2 (heads)
//                                                    score = clamp(a . e, -20, 20)
//   TransE_l1  a = h + r | t - r                     score = gamma - sum |a - e|
//   RotatE     a = x (*) rot(r) | x (*) conj(rot(r)) score = gamma - sum_k |a_k - e_k| (complex modulus),
//              rot(r) = exp(i r pi / emb_init), relations are dim / 2 phases
//
// GEMM family (TransE_l2 and the three bilinear models): the cross products a.e' over all negatives
// are ONE bf16 tensor-core GEMM over the whole batch (rs_gemm_bf16, tcgen05): S[bs, C*ns] = A . Neg^T,
// of which the chunk-diagonal blocks are consumed.  This file has the element-wise stages around it:
//   kge_prepare : a (bf16 copy for the GEMM), |a|^2, |e'|^2, positive scores, positive loss and the
//                 positive gradient of y
//   kge_neg_loss: S -> negative scores -> loss, and the weight matrix W (bf16, zero outside the
//                 chunk-diagonal) with its row / column sums for the backward GEMMs
//                 GA = W . Neg (mode 2), GB = W^T . A (mode 1)
//   kge_finish  : GA, GB -> gradients of x, r and of the negative entities
// Pairwise family (TransE_l1, RotatE): sum |a - e'| is not a contraction, so three fp32 kernels walk
// the (positive, negative) pairs of each chunk: kge_pair_forward (a warp per 4 x 4 pairs),
// kge_pair_grad_pos (four threads per element of 8 positives, sharing the chunk's negatives) and
// kge_pair_grad_neg (the transpose).  No atomics on the gradients: every output element has one owner.
#include <cuda_bf16.h>
#include "common/rs_common.h"

namespace {

enum : int { kTransE2 = 0, kDistMult = 1, kComplEx = 2, kSimplE = 3, kTransE1 = 4, kRotatE = 5, kRescal = 6 };
__host__ __device__ __forceinline__ bool is_pairwise(int model) { return model == kTransE1 || model == kRotatE; }
constexpr int kRescalCols = 16;   // columns of the relation matrix per lane: D <= 512
constexpr float kPi = 3.14159265358979323846f;

struct KgeArgs {
  const float* h; const float* r; const float* t;   // [bs, D] ([bs, Dr] for r)
  const float* neg;                                  // [C*ns, D]
  int bs, cs, ns, C, D, Dp, Dr;                      // Dp: padded row length of the bf16 operands; Dr: relation row length
  int model;
  int corrupt_head;                                  // 0: negatives replace tails, 1: heads
  float gamma, emb_init;
  __nv_bfloat16* A;                                  // [bs, Dp]
  __nv_bfloat16* Bn;                                 // [C*ns, Dp]
  float* a2; float* b2;                              // [bs], [C*ns]; a2 holds d loss / d pos score for the non-TransE_l2 models
  float* loss;                                       // [2]: positive part, negative part (already averaged and halved)
  float* gh; float* gr; float* gt;                   // gradients: [bs, D], [bs, Dr], [bs, D]
  float* gneg;                                       // [C*ns, D]
  const float* S;                                    // [bs, C*ns] cross products
  __nv_bfloat16* W;                                  // [bs, C*ns]
  float* rowsum; float* colsum;                      // [bs], [C*ns]
  const float* GA; const float* GB;                  // [bs, Dp], [C*ns, Dp]
  float* A32;                                        // pairwise family: a in fp32, [bs, Dp] (the GA buffer)
  float* Wf;                                         // pairwise family: d loss / d neg score, [bs, ns] (the S buffer)
  int vec;                                           // rows can be taken in 16-byte pieces (D, Dp and all addresses allow it)
  float* pos_score; float* neg_score;                // optional outputs (evaluation / tests): [bs], [bs, ns]
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(__expf(-fabsf(x))); }
__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }
__device__ __forceinline__ float sgn(float v) { return v > 0.f ? 1.f : (v < 0.f ? -1.f : 0.f); }

// ---- bilinear models on the element pair (k, k + D/2): a = bil(x, r) and its transpose ----------------------------
__device__ __forceinline__ void bil_fwd(int model, bool ch, float x0, float x1, float r0, float r1, float& a0, float& a1) {
  if (model == kDistMult) {
    a0 = x0 * r0; a1 = x1 * r1;
  } else if (model == kComplEx) {
    const float s = ch ? -1.f : 1.f;
    a0 = x0 * r0 - s * x1 * r1; a1 = x1 * r0 + s * x0 * r1;
  } else {  // SimplE: r0 = r, r1 = r_inv; x0 = head role, x1 = tail role
    if (!ch) { a0 = 0.5f * x1 * r1; a1 = 0.5f * x0 * r0; }
    else { a0 = 0.5f * x1 * r0; a1 = 0.5f * x0 * r1; }
  }
}
__device__ __forceinline__ void bil_bwd(int model, bool ch, float g0, float g1, float x0, float x1, float r0, float r1,
                                        float& dx0, float& dx1, float& dr0, float& dr1) {
  if (model == kDistMult) {
    dx0 = g0 * r0; dx1 = g1 * r1; dr0 = g0 * x0; dr1 = g1 * x1;
  } else if (model == kComplEx) {
    const float s = ch ? -1.f : 1.f;
    dx0 = g0 * r0 + s * g1 * r1; dx1 = g1 * r0 - s * g0 * r1;
    dr0 = g0 * x0 + g1 * x1;     dr1 = s * (g1 * x0 - g0 * x1);
  } else {
    if (!ch) { dx1 = 0.5f * g0 * r1; dr1 = 0.5f * g0 * x1; dx0 = 0.5f * g1 * r0; dr0 = 0.5f * g1 * x0; }
    else { dx1 = 0.5f * g0 * r0; dr0 = 0.5f * g0 * x1; dx0 = 0.5f * g1 * r1; dr1 = 0.5f * g1 * x0; }
  }
}

// ---- pairwise models on the element pair (k, k + D/2) -------------------------------------------------------------
// distance contribution of one pair of differences and its direction (d psi / d difference)
__device__ __forceinline__ float pair_psi(int model, float d0, float d1, float& u0, float& u1) {
  if (model == kTransE1) { u0 = sgn(d0); u1 = sgn(d1); return fabsf(d0) + fabsf(d1); }
  const float m2 = d0 * d0 + d1 * d1;
  const float inv = m2 > 0.f ? rsqrtf(m2) : 0.f;     // one special-function instruction where root and reciprocal take two
  u0 = d0 * inv; u1 = d1 * inv;
  return m2 * inv;
}
// The loops over the pairs work on TWO rows at once in packed fp32 (f32x2): they are bound by issue slots, and a packed
// instruction does the same correctly rounded operation on both halves in one slot.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// (g0, g1) += w * d psi / d difference.  RotatE: the lower bound only keeps 0 * (1 / 0) out.
__device__ __forceinline__ void pair_pull(int model, f32x2 d0, f32x2 d1, f32x2 w, f32x2& g0, f32x2& g1) {
  if (model == kTransE1) {
    float a, b;
    unpack2(d0, a, b);
    g0 = fma2(w, pack2(sgn(a), sgn(b)), g0);
    unpack2(d1, a, b);
    g1 = fma2(w, pack2(sgn(a), sgn(b)), g1);
  } else {
    float a, b;
    unpack2(fma2(d1, d1, mul2(d0, d0)), a, b);
    const f32x2 c = mul2(w, pack2(rsqrtf(fmaxf(a, 1e-37f)), rsqrtf(fmaxf(b, 1e-37f))));
    g0 = fma2(c, d0, g0);
    g1 = fma2(c, d1, g1);
  }
}
__device__ __forceinline__ f32x2 pair_dist2(int model, f32x2 d0, f32x2 d1) {
  float a, b;
  if (model == kTransE1) {
    float c, d;
    unpack2(d0, a, b);
    unpack2(d1, c, d);
    return add2(pack2(fabsf(a), fabsf(b)), pack2(fabsf(c), fabsf(d)));
  }
  unpack2(fma2(d1, d1, mul2(d0, d0)), a, b);
  return pack2(sqrtf(a), sqrtf(b));
}
__device__ __forceinline__ float pair_dist(int model, float d0, float d1) {
  return model == kTransE1 ? fabsf(d0) + fabsf(d1) : sqrtf(d0 * d0 + d1 * d1);
}

// ---- rows in 16-byte pieces (KgeArgs::vec) ---------------------------------------------------------------------------
// A warp walks a row of a few hundred floats; loads of kRowBatch pieces per lane are issued before the first is used.  (One
// element per lane and step, with stores between the loads, made the row kernels chains of a dozen memory latencies: prepare
// 12.7 us and finish 17 us for 2,048 rows of 400; now 5.7 and 5.9.)
constexpr int kRowBatch = 4;
__device__ __forceinline__ float4 add4(const float4& a, const float4& b, float s = 1.f) {
  return make_float4(a.x + s * b.x, a.y + s * b.y, a.z + s * b.z, a.w + s * b.w);
}
template <typename Load, typename Use>
__device__ __forceinline__ void for_row4(int n, int lane, Load load, Use use) {
  for (int d0 = lane * 4; d0 < n; d0 += 128 * kRowBatch) {
    decltype(load(0)) v[kRowBatch];
#pragma unroll
    for (int u = 0; u < kRowBatch; ++u)
      if (d0 + 128 * u < n) v[u] = load(d0 + 128 * u);
#pragma unroll
    for (int u = 0; u < kRowBatch; ++u)
      if (d0 + 128 * u < n) use(d0 + 128 * u, v[u]);
  }
}
// Stores four values as bf16 and returns the sum of squares of what was stored.
__device__ __forceinline__ float store_bf16x4(__nv_bfloat16* p, const float4& v) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  uint2 o;
  o.x = *reinterpret_cast<const uint32_t*>(&lo);
  o.y = *reinterpret_cast<const uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = o;
  const float2 a = __bfloat1622float2(lo), b = __bfloat1622float2(hi);
  return a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y;
}
__device__ __forceinline__ float4 load_bf16x4(const __nv_bfloat16* p) {
  const uint2 o = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// one warp per row: rows [0, bs) are positives, rows [bs, bs + C*ns) negatives
__global__ void __launch_bounds__(256) kge_prepare_kernel(const KgeArgs k) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int D = k.D, H = k.D >> 1;
  if (row >= k.bs + k.C * k.ns) return;
  if (row >= k.bs) {
    if (is_pairwise(k.model)) return;                // the pairwise kernels read the fp32 rows themselves
    const int j = row - k.bs;
    const float* src = k.neg + static_cast<size_t>(j) * D;
    __nv_bfloat16* dst = k.Bn + static_cast<size_t>(j) * k.Dp;
    float s = 0.f;
    if (k.vec) {
      for_row4(k.Dp, lane, [&](int d) { return d < D ? *reinterpret_cast<const float4*>(src + d) : make_float4(0.f, 0.f, 0.f, 0.f); },
               [&](int d, const float4& v) { s += store_bf16x4(dst + d, v); });
    } else {
      for (int d = lane; d < k.Dp; d += 32) {
        const __nv_bfloat16 b = __float2bfloat16(d < D ? src[d] : 0.f);
        dst[d] = b;
        const float vb = __bfloat162float(b);
        s += vb * vb;
      }
    }
    s = warp_sum(s);
    if (lane == 0) k.b2[j] = s;
    return;
  }
  const int i = row;
  const float* h = k.h + static_cast<size_t>(i) * D;
  const float* r = k.r + static_cast<size_t>(i) * k.Dr;
  const float* t = k.t + static_cast<size_t>(i) * D;
  float* gh = k.gh + static_cast<size_t>(i) * D;
  float* gr = k.gr + static_cast<size_t>(i) * k.Dr;
  float* gt = k.gt + static_cast<size_t>(i) * D;
  const float inv_bs = 0.5f / static_cast<float>(k.bs);

  if (k.model == kTransE2) {
    float a2 = 0.f, pos = 0.f;
    __nv_bfloat16* A = k.A + static_cast<size_t>(i) * k.Dp;
    if (k.vec) {
      for (int d0 = lane * 4; d0 < k.Dp; d0 += 128 * kRowBatch) {
        float4 hv[kRowBatch], rv[kRowBatch], tv[kRowBatch];
#pragma unroll
        for (int u = 0; u < kRowBatch; ++u) {
          const int d = d0 + 128 * u;
          const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
          hv[u] = d < D ? *reinterpret_cast<const float4*>(h + d) : z;
          rv[u] = d < D ? *reinterpret_cast<const float4*>(r + d) : z;
          tv[u] = d < D ? *reinterpret_cast<const float4*>(t + d) : z;
        }
#pragma unroll
        for (int u = 0; u < kRowBatch; ++u) {
          const int d = d0 + 128 * u;
          if (d >= k.Dp) continue;
          const float4 diff = add4(add4(hv[u], rv[u]), tv[u], -1.f);
          a2 += store_bf16x4(A + d, k.corrupt_head ? add4(tv[u], rv[u], -1.f) : add4(hv[u], rv[u]));
          pos += diff.x * diff.x + diff.y * diff.y + diff.z * diff.z + diff.w * diff.w;
        }
      }
    }
    for (int d = k.vec ? k.Dp : lane; d < k.Dp; d += 32) {
      float a = 0.f;
      if (d < D) {
        const float hv = h[d], rv = r[d], tv = t[d];
        a = k.corrupt_head ? tv - rv : hv + rv;
        const float diff = hv + rv - tv;
        pos += diff * diff;
      }
      const __nv_bfloat16 ab = __float2bfloat16(a);
      k.A[static_cast<size_t>(i) * k.Dp + d] = ab;
      const float av = __bfloat162float(ab);
      a2 += av * av;
    }
    a2 = warp_sum(a2);
    pos = warp_sum(pos);
    const float dist = sqrtf(fmaxf(pos, 1e-30f));
    const float score = k.gamma - dist;
    const float q = -sigmoid(-score) * inv_bs;      // d loss / d score of a positive
    if (lane == 0) {
      k.a2[i] = a2;
      if (k.pos_score) k.pos_score[i] = score;
      atomicAdd(&k.loss[0], -log_sigmoid(score) * inv_bs);
    }
    const float qd = -q / dist;                     // d score / d h = -(h + r - t) / dist
    if (k.vec) {
      for_row4(D, lane,
               [&](int d) {
                 return add4(add4(*reinterpret_cast<const float4*>(h + d), *reinterpret_cast<const float4*>(r + d)),
                             *reinterpret_cast<const float4*>(t + d), -1.f);
               },
               [&](int d, const float4& v) {
                 const float4 g = make_float4(qd * v.x, qd * v.y, qd * v.z, qd * v.w);
                 *reinterpret_cast<float4*>(gh + d) = g;
                 *reinterpret_cast<float4*>(gr + d) = g;
                 *reinterpret_cast<float4*>(gt + d) = make_float4(-g.x, -g.y, -g.z, -g.w);
               });
    } else {
      for (int d = lane; d < D; d += 32) {
        const float g = qd * (h[d] + r[d] - t[d]);
        gh[d] = g; gr[d] = g; gt[d] = -g;
      }
    }
    return;
  }

  const bool ch = k.corrupt_head != 0;
  const float* x = ch ? t : h;
  const float* y = ch ? h : t;
  float* gy = ch ? gh : gt;
  if (k.model == kRescal) {
    // RESCAL: score = h^T M t with one D x D matrix M per relation (row-major in r).  Tails corrupted: a = M^T h, heads
    // corrupted: a = M t; either way pos = a . y and the negatives' scores are the cross products a . e'.
    // (score_fun.py:378-449 of the reference's DGL-KE.)
    float* a32 = k.A32 + static_cast<size_t>(i) * k.Dp;   // fp32 copy of a for this kernel (the GEMM overwrites it later)
    __nv_bfloat16* A = k.A + static_cast<size_t>(i) * k.Dp;
    if (!ch) {                                        // a_j = sum_i h_i M[i][j]: every lane owns columns j = lane + 32 c
      float acc[kRescalCols];
#pragma unroll
      for (int c = 0; c < kRescalCols; ++c) acc[c] = 0.f;
      for (int row = 0; row < D; ++row) {
        const float hv = x[row];
        const float* m = r + static_cast<size_t>(row) * D;
#pragma unroll
        for (int c = 0; c < kRescalCols; ++c) {
          const int j = lane + 32 * c;
          if (j < D) acc[c] += hv * m[j];
        }
      }
#pragma unroll
      for (int c = 0; c < kRescalCols; ++c) {
        const int j = lane + 32 * c;
        if (j < D) a32[j] = acc[c];
      }
    } else {                                          // a_i = sum_j M[i][j] t_j: a row's dot product per step
      float xv[kRescalCols];
#pragma unroll
      for (int c = 0; c < kRescalCols; ++c) {
        const int j = lane + 32 * c;
        xv[c] = j < D ? x[j] : 0.f;
      }
      for (int row = 0; row < D; ++row) {
        const float* m = r + static_cast<size_t>(row) * D;
        float p = 0.f;
#pragma unroll
        for (int c = 0; c < kRescalCols; ++c) {
          const int j = lane + 32 * c;
          if (j < D) p += m[j] * xv[c];
        }
        p = warp_sum(p);
        if (lane == 0) a32[row] = p;
      }
    }
    __syncwarp();
    float pos = 0.f;
    for (int d = lane; d < k.Dp; d += 32) {
      const float a = d < D ? a32[d] : 0.f;
      A[d] = __float2bfloat16(a);
      if (d < D) pos += a * y[d];
    }
    pos = warp_sum(pos);
    const float q = -sigmoid(-pos) * inv_bs;
    if (lane == 0) {
      k.a2[i] = q;
      if (k.pos_score) k.pos_score[i] = pos;
      atomicAdd(&k.loss[0], -log_sigmoid(pos) * inv_bs);
    }
    for (int d = lane; d < D; d += 32) gy[d] = q * a32[d];
    return;
  }
  if (k.model <= kSimplE) {                           // bilinear: a = bil(x, r), pos = a . y
    float pos = 0.f;
    __nv_bfloat16* A = k.A + static_cast<size_t>(i) * k.Dp;
    for (int kk = lane; kk < H; kk += 32) {
      float a0, a1;
      bil_fwd(k.model, ch, x[kk], x[kk + H], r[kk], r[kk + H], a0, a1);
      A[kk] = __float2bfloat16(a0); A[kk + H] = __float2bfloat16(a1);
      pos += a0 * y[kk] + a1 * y[kk + H];
    }
    for (int d = D + lane; d < k.Dp; d += 32) A[d] = __float2bfloat16(0.f);
    pos = warp_sum(pos);
    float score = pos, pass = 1.f;
    if (k.model == kSimplE) { score = fminf(fmaxf(pos, -20.f), 20.f); pass = (pos >= -20.f && pos <= 20.f) ? 1.f : 0.f; }
    const float q = -sigmoid(-score) * inv_bs * pass;
    if (lane == 0) {
      k.a2[i] = q;
      if (k.pos_score) k.pos_score[i] = score;
      atomicAdd(&k.loss[0], -log_sigmoid(score) * inv_bs);
    }
    for (int kk = lane; kk < H; kk += 32) {          // d pos / d y = a (recomputed in fp32)
      float a0, a1;
      bil_fwd(k.model, ch, x[kk], x[kk + H], r[kk], r[kk + H], a0, a1);
      gy[kk] = q * a0; gy[kk + H] = q * a1;
    }
    return;
  }

  // pairwise: a in fp32 for the pair kernels, pos = gamma - sum psi(a - y)
  const float sg = ch ? -1.f : 1.f;
  const float to_phase = kPi / k.emb_init;
  float* A32 = k.A32 + static_cast<size_t>(i) * k.Dp;
  float dist = 0.f;
  const bool l1 = k.model == kTransE1;
  for (int kk0 = lane; kk0 < H; kk0 += 32 * kRowBatch) {           // loads of kRowBatch elements before the first is used
    float x0[kRowBatch], x1[kRowBatch], y0[kRowBatch], y1[kRowBatch], r0[kRowBatch], r1[kRowBatch];
#pragma unroll
    for (int u = 0; u < kRowBatch; ++u) {
      const int kk = min(kk0 + 32 * u, H - 1);
      x0[u] = x[kk]; x1[u] = x[kk + H]; y0[u] = y[kk]; y1[u] = y[kk + H];
      r0[u] = r[kk]; r1[u] = l1 ? r[kk + H] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kRowBatch; ++u) {
      const int kk = kk0 + 32 * u;
      if (kk >= H) break;
      float a0, a1;
      if (l1) {
        a0 = x0[u] + sg * r0[u]; a1 = x1[u] + sg * r1[u];
      } else {
        float sn, c;
        __sincosf(r0[u] * to_phase, &sn, &c);
        a0 = x0[u] * c - sg * x1[u] * sn; a1 = sg * x0[u] * sn + x1[u] * c;
      }
      A32[kk] = a0; A32[kk + H] = a1;
      dist += pair_dist(k.model, a0 - y0[u], a1 - y1[u]);
    }
  }
  dist = warp_sum(dist);
  const float score = k.gamma - dist;
  const float q = -sigmoid(-score) * inv_bs;
  if (lane == 0) {
    k.a2[i] = q;
    if (k.pos_score) k.pos_score[i] = score;
    atomicAdd(&k.loss[0], -log_sigmoid(score) * inv_bs);
  }
  for (int kk0 = lane; kk0 < H; kk0 += 32 * kRowBatch) {           // d loss / d y = q * (-1) * (-u)
    float d0[kRowBatch], d1[kRowBatch];
#pragma unroll
    for (int u = 0; u < kRowBatch; ++u) {
      const int kk = min(kk0 + 32 * u, H - 1);
      d0[u] = A32[kk] - y[kk]; d1[u] = A32[kk + H] - y[kk + H];
    }
#pragma unroll
    for (int u = 0; u < kRowBatch; ++u) {
      const int kk = kk0 + 32 * u;
      if (kk >= H) break;
      float u0, u1;
      pair_psi(k.model, d0[u], d1[u], u0, u1);
      gy[kk] = q * u0; gy[kk + H] = q * u1;
    }
  }
}

// W row-major [bs, C*ns], zero outside the chunk diagonal.  A block takes 8 positives (one per warp) x 256 columns, a lane 8
// neighbouring columns: row sums leave with one atomic per warp, column sums meet in shared memory over the 8 rows and leave
// with one atomic per column, the loss with one per block.  (A thread per element with two global atomics each spent 37 us
// on 524,288 atomics for 1,024 x 256 pairs, this form 6; a block off the diagonal only writes zeros.)
constexpr int kLossCols = 256;
__global__ void __launch_bounds__(256) kge_neg_loss_kernel(const KgeArgs k) {
  __shared__ float s_w[8][kLossCols];
  __shared__ float s_l[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ncols = k.C * k.ns;
  const int i = blockIdx.y * 8 + warp;
  const int c0 = blockIdx.x * kLossCols;
  const int col = c0 + lane * 8;                      // (ncols is a multiple of 8: the GEMM asks for it)
  const bool row_ok = i < k.bs;
  const int c = row_ok ? i / k.cs : 0;
  const int lo = c * k.ns, hi = lo + k.ns;            // the columns of this row's chunk
  float w[8], l = 0.f, rs = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = 0.f;
  if (row_ok && col < hi && col + 8 > lo && col < ncols) {
    const float* sp = k.S + static_cast<size_t>(i) * ncols + col;
    const float4 s0 = *reinterpret_cast<const float4*>(sp), s1 = *reinterpret_cast<const float4*>(sp + 4);
    const float dot[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    const float norm = 1.f / (static_cast<float>(k.bs) * k.ns) * 0.5f;
    const float a2 = k.model == kTransE2 ? k.a2[i] : 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (col + e < lo || col + e >= hi) continue;
      float score, wgt;
      if (k.model == kTransE2) {
        const float dist = sqrtf(fmaxf(a2 + k.b2[col + e] - 2.f * dot[e], 1e-30f));
        score = k.gamma - dist;
        wgt = sigmoid(score) * norm / dist;      // q / dist
      } else if (k.model == kSimplE) {
        score = fminf(fmaxf(dot[e], -20.f), 20.f);
        wgt = (dot[e] >= -20.f && dot[e] <= 20.f) ? sigmoid(score) * norm : 0.f;
      } else {
        score = dot[e];
        wgt = sigmoid(score) * norm;             // q
      }
      l -= log_sigmoid(-score) * norm;
      if (k.neg_score) k.neg_score[static_cast<size_t>(i) * k.ns + (col + e - lo)] = score;
      w[e] = __bfloat162float(__float2bfloat16(wgt));
      rs += w[e];
    }
  }
  if (row_ok && col < ncols) {
    uint4 o;
    __nv_bfloat16* oe = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
    for (int e = 0; e < 8; ++e) oe[e] = __float2bfloat16(w[e]);
    *reinterpret_cast<uint4*>(k.W + static_cast<size_t>(i) * ncols + col) = o;
  }
  // off the diagonal for all of the block's rows: zeros are written, nothing is left to add
  const int first = blockIdx.y * 8, last = min(k.bs, first + 8) - 1;
  if (c0 >= (last / k.cs + 1) * k.ns || c0 + kLossCols <= (first / k.cs) * k.ns) return;
  rs = warp_sum(rs);
  l = warp_sum(l);
  if (lane == 0) {
    if (row_ok && rs != 0.f) atomicAdd(&k.rowsum[i], rs);
    s_l[warp] = l;
  }
  *reinterpret_cast<float4*>(&s_w[warp][lane * 8]) = make_float4(w[0], w[1], w[2], w[3]);
  *reinterpret_cast<float4*>(&s_w[warp][lane * 8 + 4]) = make_float4(w[4], w[5], w[6], w[7]);
  __syncthreads();
  const int my = c0 + threadIdx.x;
  float cs = 0.f;
#pragma unroll
  for (int q = 0; q < 8; ++q) cs += s_w[q][threadIdx.x];
  if (my < ncols && cs != 0.f) atomicAdd(&k.colsum[my], cs);
  if (threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += s_l[q];
    if (t != 0.f) atomicAdd(&k.loss[1], t);
  }
}

// one warp per row again
__global__ void __launch_bounds__(256) kge_finish_kernel(const KgeArgs k) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int D = k.D, H = k.D >> 1;
  if (row >= k.bs + k.C * k.ns) return;
  if (row >= k.bs) {
    const int j = row - k.bs;
    const float cs = k.model == kTransE2 ? k.colsum[j] : 0.f;
    if (k.vec) {
      const float* gb = k.GB + static_cast<size_t>(j) * k.Dp;
      const __nv_bfloat16* bn = k.Bn + static_cast<size_t>(j) * k.Dp;
      float* out = k.gneg + static_cast<size_t>(j) * D;
      const bool centred = k.model == kTransE2;
      for_row4(D, lane,
               [&](int d) {
                 const float4 g = *reinterpret_cast<const float4*>(gb + d);
                 return centred ? add4(g, load_bf16x4(bn + d), -cs) : g;
               },
               [&](int d, const float4& g) { *reinterpret_cast<float4*>(out + d) = g; });
      return;
    }
    for (int d = lane; d < D; d += 32) {
      float g = k.GB[static_cast<size_t>(j) * k.Dp + d];
      if (k.model == kTransE2) g -= cs * __bfloat162float(k.Bn[static_cast<size_t>(j) * k.Dp + d]);
      k.gneg[static_cast<size_t>(j) * D + d] = g;
    }
    return;
  }
  const int i = row;
  float* gh = k.gh + static_cast<size_t>(i) * D;
  float* gr = k.gr + static_cast<size_t>(i) * k.Dr;
  float* gt = k.gt + static_cast<size_t>(i) * D;
  const float* GA = k.GA + static_cast<size_t>(i) * k.Dp;
  if (k.model == kTransE2) {
    const float rs = k.rowsum[i];
    if (k.vec) {
      const __nv_bfloat16* A = k.A + static_cast<size_t>(i) * k.Dp;
      float* gx = k.corrupt_head ? gt : gh;                   // a = t - r  or  a = h + r
      const float sr = k.corrupt_head ? -1.f : 1.f;
      for (int d0 = lane * 4; d0 < D; d0 += 128 * kRowBatch) {
        float4 ga[kRowBatch], x[kRowBatch], r[kRowBatch];
#pragma unroll
        for (int u = 0; u < kRowBatch; ++u) {
          const int d = d0 + 128 * u;
          if (d >= D) continue;
          ga[u] = add4(*reinterpret_cast<const float4*>(GA + d), load_bf16x4(A + d), -rs);
          x[u] = *reinterpret_cast<const float4*>(gx + d);
          r[u] = *reinterpret_cast<const float4*>(gr + d);
        }
#pragma unroll
        for (int u = 0; u < kRowBatch; ++u) {
          const int d = d0 + 128 * u;
          if (d >= D) continue;
          *reinterpret_cast<float4*>(gx + d) = add4(x[u], ga[u]);
          *reinterpret_cast<float4*>(gr + d) = add4(r[u], ga[u], sr);
        }
      }
      return;
    }
    for (int d = lane; d < D; d += 32) {
      const float ga = GA[d] - rs * __bfloat162float(k.A[static_cast<size_t>(i) * k.Dp + d]);
      if (k.corrupt_head) { gt[d] += ga; gr[d] -= ga; }    // a = t - r
      else { gh[d] += ga; gr[d] += ga; }                   // a = h + r
    }
    return;
  }
  if (k.model == kRescal) {
    // g = d loss / d a = q * y + GA.  Tails corrupted (a = M^T h): dh = M g, dM[i][j] = h_i g_j.  Heads corrupted
    // (a = M t): dt = M^T g, dM[i][j] = g_i t_j.  rowsum[i] receives |dM|^2 = |g|^2 |x|^2, the squared norm of this
    // occurrence's whole matrix gradient: the row-blocked relation table turns it into ONE Adagrad state per relation.
    const bool chr = k.corrupt_head != 0;
    const float* x = (chr ? k.t : k.h) + static_cast<size_t>(i) * D;
    const float* y = (chr ? k.h : k.t) + static_cast<size_t>(i) * D;
    const float* M = k.r + static_cast<size_t>(i) * k.Dr;
    float* gx = chr ? gt : gh;
    float* g = const_cast<float*>(GA);               // this kernel is the last reader of GA: g is formed in place
    const float q = k.a2[i];
    float g2 = 0.f, x2 = 0.f;
    for (int d = lane; d < D; d += 32) {
      const float gv = q * y[d] + GA[d];
      g[d] = gv;
      g2 += gv * gv;
      x2 += x[d] * x[d];
    }
    g2 = warp_sum(g2);
    x2 = warp_sum(x2);
    if (lane == 0) k.rowsum[i] = g2 * x2;
    __syncwarp();
    float gv[kRescalCols], xv[kRescalCols], acc[kRescalCols];
#pragma unroll
    for (int c = 0; c < kRescalCols; ++c) {
      const int j = lane + 32 * c;
      gv[c] = j < D ? g[j] : 0.f;
      xv[c] = j < D ? x[j] : 0.f;
      acc[c] = 0.f;
    }
    for (int row = 0; row < D; ++row) {
      const float* m = M + static_cast<size_t>(row) * D;
      float* dm = gr + static_cast<size_t>(row) * D;
      if (!chr) {                                     // dh_row = M[row,:] . g ; dM[row][j] = h_row g_j
        const float hv = x[row];
        float p = 0.f;
#pragma unroll
        for (int c = 0; c < kRescalCols; ++c) {
          const int j = lane + 32 * c;
          if (j < D) { p += m[j] * gv[c]; dm[j] = hv * gv[c]; }
        }
        p = warp_sum(p);
        if (lane == 0) gx[row] = p;
      } else {                                        // dt_j += g_row M[row][j] ; dM[row][j] = g_row t_j
        const float gr_ = g[row];
#pragma unroll
        for (int c = 0; c < kRescalCols; ++c) {
          const int j = lane + 32 * c;
          if (j < D) { acc[c] += gr_ * m[j]; dm[j] = gr_ * xv[c]; }
        }
      }
    }
    if (chr) {
#pragma unroll
      for (int c = 0; c < kRescalCols; ++c) {
        const int j = lane + 32 * c;
        if (j < D) gx[j] = acc[c];
      }
    }
    return;
  }
  // bilinear: d loss / d a = q * y (positive) + GA (negatives); chain through a = bil(x, r)
  const bool ch = k.corrupt_head != 0;
  const float* x = (ch ? k.t : k.h) + static_cast<size_t>(i) * D;
  const float* y = (ch ? k.h : k.t) + static_cast<size_t>(i) * D;
  const float* r = k.r + static_cast<size_t>(i) * k.Dr;
  float* gx = ch ? gt : gh;
  const float q = k.a2[i];
  for (int kk = lane; kk < H; kk += 32) {
    const float g0 = q * y[kk] + GA[kk], g1 = q * y[kk + H] + GA[kk + H];
    float dx0, dx1, dr0, dr1;
    bil_bwd(k.model, ch, g0, g1, x[kk], x[kk + H], r[kk], r[kk + H], dx0, dx1, dr0, dr1);
    gx[kk] = dx0; gx[kk + H] = dx1; gr[kk] = dr0; gr[kk + H] = dr1;
  }
}

// ---- pairwise family ---------------------------------------------------------------------------------------------
// A warp scores 4 positives against 4 negatives of their chunk: every lane strides over the element pairs and keeps
// 16 partial distances, which a transposing butterfly reduces so that lanes 2 p and 2 p + 1 end with pair p = (p / 4, p % 4).
// Bound by latency and issue slots, operands come from L1 / L2: 16 sums leave room for twice the warps that 4 x 8 pairs did
// (114 registers, 23 % of the warps resident, 53 us for 1,024 x 256 pairs of 200 complex elements; now 37 us).
constexpr int kPairTileI = 4, kPairTileJ = 4;
template <int MODEL>
__global__ void __launch_bounds__(256, 3) kge_pair_forward_kernel(const KgeArgs k) {
  __shared__ float s_l[8];
  const int lane = threadIdx.x & 31;
  const int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int jt = k.ns / kPairTileJ;                // tiles of negatives per chunk
  const int n_warps = (k.bs / kPairTileI) * jt;
  float l = 0.f;
  if (warp < n_warps) {
    const int i0 = (warp / jt) * kPairTileI, j0 = (warp % jt) * kPairTileJ;
    const int c = i0 / k.cs;
    const int H = k.D >> 1;
    const float* a = k.A32 + static_cast<size_t>(i0) * k.Dp;
    const float* n = k.neg + (static_cast<size_t>(c) * k.ns + j0) * k.D;
    f32x2 v2[2][4];                                // positives 2 q and 2 q + 1 against negative jj
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) v2[q][jj] = 0ull;
    // The operands of the next step are fetched while this one's pairs are worked out; past the end the last are fetched again.
    float a0[4], a1[4], n0[4], n1[4];
    auto fetch = [&](int kk) {
      kk = min(kk, H - 1);
#pragma unroll
      for (int ii = 0; ii < 4; ++ii) { a0[ii] = a[ii * k.Dp + kk]; a1[ii] = a[ii * k.Dp + kk + H]; }
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) { n0[jj] = n[jj * k.D + kk]; n1[jj] = n[jj * k.D + kk + H]; }
    };
    fetch(lane);
    for (int kk = lane; kk < H; kk += 32) {
      f32x2 b0[2], b1[2], m0[4], m1[4];
#pragma unroll
      for (int q = 0; q < 2; ++q) { b0[q] = pack2(a0[2 * q], a0[2 * q + 1]); b1[q] = pack2(a1[2 * q], a1[2 * q + 1]); }
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) { m0[jj] = pack2(-n0[jj], -n0[jj]); m1[jj] = pack2(-n1[jj], -n1[jj]); }
      fetch(kk + 32);
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) v2[q][jj] = add2(v2[q][jj], pair_dist2(MODEL, add2(b0[q], m0[jj]), add2(b1[q], m1[jj])));
    }
    float v[16];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) unpack2(v2[q][jj], v[8 * q + jj], v[8 * q + 4 + jj]);
#pragma unroll
    for (int o = 16, cnt = 16; o > 1; o >>= 1, cnt >>= 1) {
      const bool upper = (lane & o) != 0;
#pragma unroll
      for (int p = 0; p < cnt / 2; ++p) {
        const float send = upper ? v[p] : v[p + cnt / 2];
        const float keep = upper ? v[p + cnt / 2] : v[p];
        v[p] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    if ((lane & 1) == 0) {
      const int p = lane >> 1;
      const int i = i0 + (p >> 2), j = j0 + (p & 3);
      const float score = k.gamma - v[0];
      const float norm = 1.f / (static_cast<float>(k.bs) * k.ns) * 0.5f;
      k.Wf[static_cast<size_t>(i) * k.ns + j] = sigmoid(score) * norm;     // d loss / d score
      if (k.neg_score) k.neg_score[static_cast<size_t>(i) * k.ns + j] = score;
      l = -log_sigmoid(-score) * norm;
    }
  }
  // one atomic per block: a chain of fewer and larger terms is also the more exact sum
  l = warp_sum(l);
  if (lane == 0) s_l[threadIdx.x >> 5] = l;
  __syncthreads();
  if (threadIdx.x == 0) {
    l = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) l += s_l[q];
    if (l != 0.f) atomicAdd(&k.loss[1], l);
  }
}

constexpr int kPairRows = 8;      // rows that share one pass over the other side
constexpr int kPairTile = 256;    // weights staged per pass
constexpr int kPairCols = 32;     // element pairs per block: a warp per way
constexpr int kPairWays = 4;      // warps that share an element pair, each walking its part of the other side
constexpr int kPairThreads = kPairCols * kPairWays;
constexpr int kPairBatch = 2;     // rows of the other side a thread fetches at once

// Sums the kPairWays partial gradients of every element pair into the threads of way 0.
__device__ __forceinline__ void pair_join(f32x2 (&g0)[kPairRows / 2], f32x2 (&g1)[kPairRows / 2], float* mem, int col, int way) {
  f32x2* buf = reinterpret_cast<f32x2*>(mem);
  for (int q = 1; q < kPairWays; ++q) {
    __syncthreads();
    if (way == q) {
#pragma unroll
      for (int rr = 0; rr < kPairRows / 2; ++rr) {
        buf[(2 * rr) * kPairCols + col] = g0[rr];
        buf[(2 * rr + 1) * kPairCols + col] = g1[rr];
      }
    }
    __syncthreads();
    if (way == 0) {
#pragma unroll
      for (int rr = 0; rr < kPairRows / 2; ++rr) {
        g0[rr] = add2(g0[rr], buf[(2 * rr) * kPairCols + col]);
        g1[rr] = add2(g1[rr], buf[(2 * rr + 1) * kPairCols + col]);
      }
    }
  }
}

// The two gradient kernels: a block owns 8 rows of one side x 32 element pairs; its 4 warps walk a quarter of the
// other side's rows of the chunk each and add up at the end, so every gradient element still has one owner and no atomics.
// Bound by the latency of the other side's rows; one way of 128 threads left three quarters of the warps out: 167 and 159 us
// for 1,024 x 256 pairs of 200 complex elements, 9 % resident.  Now 48 and 45 us, of which the special-function unit accounts
// for 12; fetching four rows at a time instead of two cost registers and was slower (75 and 67 us).

// Block = 8 positives of one chunk; chains d loss / d a (negatives and the positive) to x and r.
template <int MODEL>
__global__ void __launch_bounds__(kPairThreads, 8) kge_pair_grad_pos_kernel(const KgeArgs k) {
  __shared__ __align__(16) float w[kPairTile][kPairRows];      // (the join's 8 x 32 packed pairs fit into it)
  const int i0 = blockIdx.x * kPairRows;
  const int c = i0 / k.cs;
  const int H = k.D >> 1;
  const int col = threadIdx.x % kPairCols, way = threadIdx.x / kPairCols;
  const int kk = blockIdx.y * kPairCols + col;
  const bool live = kk < H;
  f32x2 a0[kPairRows / 2], a1[kPairRows / 2], g0[kPairRows / 2], g1[kPairRows / 2];   // rows 2 q and 2 q + 1
#pragma unroll
  for (int q = 0; q < kPairRows / 2; ++q) {
    const float* lo = k.A32 + static_cast<size_t>(i0 + 2 * q) * k.Dp;
    const float* hi = lo + k.Dp;
    a0[q] = live ? pack2(lo[kk], hi[kk]) : 0ull;
    a1[q] = live ? pack2(lo[kk + H], hi[kk + H]) : 0ull;
    g0[q] = 0ull; g1[q] = 0ull;
  }
  for (int jb = 0; jb < k.ns; jb += kPairTile) {
    const int nj = min(kPairTile, k.ns - jb);
    __syncthreads();
    for (int e = threadIdx.x; e < kPairRows * nj; e += kPairThreads) {
      const int rr = e / nj, j = e - rr * nj;
      w[j][rr] = k.Wf[static_cast<size_t>(i0 + rr) * k.ns + jb + j];
    }
    __syncthreads();
    if (live) {
      const float* n = k.neg + (static_cast<size_t>(c) * k.ns + jb) * k.D + kk;
      // kPairBatch rows of the other side are fetched together
      for (int jj0 = way; jj0 < nj; jj0 += kPairWays * kPairBatch) {
        float n0[kPairBatch], n1[kPairBatch];
#pragma unroll
        for (int q = 0; q < kPairBatch; ++q) {
          const float* p = n + static_cast<size_t>(min(jj0 + q * kPairWays, nj - 1)) * k.D;
          n0[q] = p[0]; n1[q] = p[H];
        }
#pragma unroll
        for (int q = 0; q < kPairBatch; ++q) {
          const int j = jj0 + q * kPairWays;
          if (j >= nj) break;
          const ulonglong2 wa = *reinterpret_cast<const ulonglong2*>(&w[j][0]), wb = *reinterpret_cast<const ulonglong2*>(&w[j][4]);
          const f32x2 ww[kPairRows / 2] = {wa.x, wa.y, wb.x, wb.y};
          const f32x2 m0 = pack2(-n0[q], -n0[q]), m1 = pack2(-n1[q], -n1[q]);
#pragma unroll
          for (int rr = 0; rr < kPairRows / 2; ++rr) pair_pull(MODEL, add2(a0[rr], m0), add2(a1[rr], m1), ww[rr], g0[rr], g1[rr]);
        }
      }
    }
  }
  pair_join(g0, g1, &w[0][0], col, way);
  if (!live || way != 0) return;
  const bool ch = k.corrupt_head != 0;
  const float sg = ch ? -1.f : 1.f;
  const float to_phase = kPi / k.emb_init;
#pragma unroll
  for (int rr = 0; rr < kPairRows; ++rr) {
    const int i = i0 + rr;
    const float* x = (ch ? k.t : k.h) + static_cast<size_t>(i) * k.D;
    const float* y = (ch ? k.h : k.t) + static_cast<size_t>(i) * k.D;
    float* gx = (ch ? k.gt : k.gh) + static_cast<size_t>(i) * k.D;
    float* gr = k.gr + static_cast<size_t>(i) * k.Dr;
    float u0, u1, p0[2], p1[2], s0[2], s1[2];
    unpack2(a0[rr / 2], p0[0], p0[1]);
    unpack2(a1[rr / 2], p1[0], p1[1]);
    unpack2(g0[rr / 2], s0[0], s0[1]);
    unpack2(g1[rr / 2], s1[0], s1[1]);
    pair_psi(MODEL, p0[rr & 1] - y[kk], p1[rr & 1] - y[kk + H], u0, u1);
    const float q = k.a2[i];
    const float ga0 = -s0[rr & 1] - q * u0, ga1 = -s1[rr & 1] - q * u1;     // (d loss / d dist = -w)
    if (MODEL == kTransE1) {
      gx[kk] = ga0; gx[kk + H] = ga1; gr[kk] = sg * ga0; gr[kk + H] = sg * ga1;
    } else {
      float sn, cs_;
      __sincosf(k.r[static_cast<size_t>(i) * k.Dr + kk] * to_phase, &sn, &cs_);
      const float x0 = x[kk], x1 = x[kk + H];
      gx[kk] = ga0 * cs_ + sg * ga1 * sn;
      gx[kk + H] = ga1 * cs_ - sg * ga0 * sn;
      const float dc = ga0 * x0 + ga1 * x1, ds = sg * (ga1 * x0 - ga0 * x1);
      gr[kk] = (ds * cs_ - dc * sn) * to_phase;
    }
  }
}

// Block = 8 negatives of one chunk; its threads walk the chunk's positives.
template <int MODEL>
__global__ void __launch_bounds__(kPairThreads, 8) kge_pair_grad_neg_kernel(const KgeArgs k) {
  __shared__ __align__(16) float w[kPairTile][kPairRows];
  const int col0 = blockIdx.x * kPairRows;          // index into [C*ns]
  const int c = col0 / k.ns, j0 = col0 - c * k.ns;
  const int H = k.D >> 1;
  const int col = threadIdx.x % kPairCols, way = threadIdx.x / kPairCols;
  const int kk = blockIdx.y * kPairCols + col;
  const bool live = kk < H;
  f32x2 n0[kPairRows / 2], n1[kPairRows / 2], g0[kPairRows / 2], g1[kPairRows / 2];   // minus rows 2 q and 2 q + 1
#pragma unroll
  for (int q = 0; q < kPairRows / 2; ++q) {
    const float* lo = k.neg + static_cast<size_t>(col0 + 2 * q) * k.D;
    const float* hi = lo + k.D;
    n0[q] = live ? pack2(-lo[kk], -hi[kk]) : 0ull;
    n1[q] = live ? pack2(-lo[kk + H], -hi[kk + H]) : 0ull;
    g0[q] = 0ull; g1[q] = 0ull;
  }
  for (int ib = 0; ib < k.cs; ib += kPairTile) {
    const int ni = min(kPairTile, k.cs - ib);
    __syncthreads();
    for (int e = threadIdx.x; e < ni * kPairRows; e += kPairThreads) {
      const int ii = e / kPairRows, jj = e - ii * kPairRows;
      w[ii][jj] = k.Wf[static_cast<size_t>(c * k.cs + ib + ii) * k.ns + j0 + jj];
    }
    __syncthreads();
    if (live) {
      const float* a = k.A32 + static_cast<size_t>(c * k.cs + ib) * k.Dp + kk;
      for (int ii0 = way; ii0 < ni; ii0 += kPairWays * kPairBatch) {
        float a0[kPairBatch], a1[kPairBatch];
#pragma unroll
        for (int q = 0; q < kPairBatch; ++q) {
          const float* p = a + static_cast<size_t>(min(ii0 + q * kPairWays, ni - 1)) * k.Dp;
          a0[q] = p[0]; a1[q] = p[H];
        }
#pragma unroll
        for (int q = 0; q < kPairBatch; ++q) {
          const int ii = ii0 + q * kPairWays;
          if (ii >= ni) break;
          const ulonglong2 wa = *reinterpret_cast<const ulonglong2*>(&w[ii][0]), wb = *reinterpret_cast<const ulonglong2*>(&w[ii][4]);
          const f32x2 ww[kPairRows / 2] = {wa.x, wa.y, wb.x, wb.y};
          const f32x2 p0 = pack2(a0[q], a0[q]), p1 = pack2(a1[q], a1[q]);
#pragma unroll
          for (int jj = 0; jj < kPairRows / 2; ++jj)      // d loss / d dist = -w, d dist / d e' = -u
            pair_pull(MODEL, add2(p0, n0[jj]), add2(p1, n1[jj]), ww[jj], g0[jj], g1[jj]);
        }
      }
    }
  }
  pair_join(g0, g1, &w[0][0], col, way);
  if (!live || way != 0) return;
#pragma unroll
  for (int q = 0; q < kPairRows / 2; ++q) {
    float* lo = k.gneg + static_cast<size_t>(col0 + 2 * q) * k.D;
    float* hi = lo + k.D;
    unpack2(g0[q], lo[kk], hi[kk]);
    unpack2(g1[q], lo[kk + H], hi[kk + H]);
  }
}

}  // namespace

// stage: 0 prepare, 1 negative loss, 2 finish.  model: 0 TransE_l2, 1 DistMult, 2 ComplEx, 3 SimplE (these four
// have the GEMMs S = A.Bn^T between stages 0 and 1 and GA = W.Bn, GB = W^T.A between 1 and 2), 4 TransE_l1,
// 5 RotatE (no GEMM: stage 1 and 2 walk the pairs; GA doubles as the fp32 copy of a, S as the pair weights), 6 RESCAL
// (GEMM family; r holds a row-major D x D matrix per positive, gr receives its gradient, rowsum the squared norm of it).
RS_API int rs_kge_stage(int stage, const float* h, const float* r, const float* t, const float* neg, int bs, int cs, int ns,
                        int D, int Dp, int Dr, int model, int corrupt_head, float gamma, float emb_init, void* A, void* Bn,
                        float* a2, float* b2, float* loss, float* gh, float* gr, float* gt, float* gneg, float* S, void* W,
                        float* rowsum, float* colsum, float* GA, const float* GB, float* pos_score, float* neg_score,
                        cudaStream_t stream) {
  RS_REQUIRE(bs > 0 && cs > 0 && bs % cs == 0 && ns > 0 && D > 0 && Dp >= D, "rs_kge_stage: bad sizes");
  RS_REQUIRE(model >= kTransE2 && model <= kRescal, "rs_kge_stage: model must be 0..6");
  RS_REQUIRE(model == kTransE2 || D % 2 == 0, "rs_kge_stage: this model splits the embedding into two halves");
  RS_REQUIRE(Dr == (model == kRotatE ? D / 2 : model == kRescal ? D * D : D), "rs_kge_stage: relation row length");
  RS_REQUIRE(model != kRescal || D <= 32 * kRescalCols, "rs_kge_stage: RESCAL needs dim <= 512");
  const bool pairwise = is_pairwise(model);
  RS_REQUIRE(!pairwise || (cs % kPairRows == 0 && ns % kPairRows == 0 && emb_init > 0.f),
             "rs_kge_stage: TransE_l1 / RotatE need chunk and negative counts that are multiples of 8");
  KgeArgs k;
  k.h = h; k.r = r; k.t = t; k.neg = neg; k.bs = bs; k.cs = cs; k.ns = ns; k.C = bs / cs; k.D = D; k.Dp = Dp; k.Dr = Dr;
  k.model = model; k.corrupt_head = corrupt_head; k.gamma = gamma; k.emb_init = emb_init;
  k.A = reinterpret_cast<__nv_bfloat16*>(A); k.Bn = reinterpret_cast<__nv_bfloat16*>(Bn); k.a2 = a2; k.b2 = b2; k.loss = loss;
  k.gh = gh; k.gr = gr; k.gt = gt; k.gneg = gneg; k.S = S; k.W = reinterpret_cast<__nv_bfloat16*>(W);
  k.rowsum = rowsum; k.colsum = colsum; k.GA = GA; k.GB = GB; k.A32 = GA; k.Wf = S;
  k.pos_score = pos_score; k.neg_score = neg_score;
  uintptr_t bits = 0;
  const void* const rows16[] = {h, r, t, neg, gh, gr, gt, gneg, GA, GB, A, Bn};
  for (const void* q : rows16) bits |= reinterpret_cast<uintptr_t>(q);
  k.vec = D % 4 == 0 && Dp % 8 == 0 && (bits & 15) == 0;
  const int rows = bs + k.C * ns;
  const int H = D / 2;
  if (stage == 0) {
    kge_prepare_kernel<<<((pairwise ? bs : rows) + 7) / 8, 256, 0, stream>>>(k);
  } else if (stage == 1) {
    if (pairwise) {
      const int warps = (bs / kPairTileI) * (ns / kPairTileJ);
      if (model == kTransE1) kge_pair_forward_kernel<kTransE1><<<(warps + 7) / 8, 256, 0, stream>>>(k);
      else kge_pair_forward_kernel<kRotatE><<<(warps + 7) / 8, 256, 0, stream>>>(k);
    } else {
      RS_REQUIRE((k.C * ns) % 8 == 0, "rs_kge_stage: the number of negatives (%d) must be a multiple of 8", k.C * ns);
      kge_neg_loss_kernel<<<dim3((k.C * ns + kLossCols - 1) / kLossCols, (bs + 7) / 8), 256, 0, stream>>>(k);
    }
  } else if (stage == 2) {
    if (pairwise) {
      const dim3 gp(bs / kPairRows, (H + kPairCols - 1) / kPairCols);
      if (model == kTransE1) kge_pair_grad_pos_kernel<kTransE1><<<gp, kPairThreads, 0, stream>>>(k);
      else kge_pair_grad_pos_kernel<kRotatE><<<gp, kPairThreads, 0, stream>>>(k);
      RS_LAUNCH_CHECK();
      const dim3 gn(k.C * ns / kPairRows, (H + kPairCols - 1) / kPairCols);
      if (model == kTransE1) kge_pair_grad_neg_kernel<kTransE1><<<gn, kPairThreads, 0, stream>>>(k);
      else kge_pair_grad_neg_kernel<kRotatE><<<gn, kPairThreads, 0, stream>>>(k);
    } else {
      kge_finish_kernel<<<(rows + 7) / 8, 256, 0, stream>>>(k);
    }
  } else {
    return rs::set_error(RS_ERR_INVALID, "rs_kge_stage: unknown stage %d", stage);
  }
  RS_LAUNCH_CHECK();
  return RS_OK;
}
