// Row access in units of V floats (V = 8: 32 bytes per lane, V = 4: 16 bytes) and the lane geometry that goes with it.
//
// A row of D floats is handled by a sub-warp of L lanes, each holding NC units, so a 32-float row occupies 4 lanes and not a
// warp of which 24 idle, and a 128-float row half a warp.  The row kernels are bound by issue slots and by the number of rows
// in flight, not by DRAM, on the skewed id streams of real use (most rows come from L2), so lanes that idle cost time.
#pragma once
#include <cuda_bf16.h>
#include <cstdint>

namespace rs {

template <int V> struct RowVec { float v[V]; };

__device__ __forceinline__ void row_load_nc(RowVec<8>& r, const float* p) {
  asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]), "=f"(r.v[4]), "=f"(r.v[5]), "=f"(r.v[6]), "=f"(r.v[7])
               : "l"(p));
}
__device__ __forceinline__ void row_load_nc(RowVec<4>& r, const float* p) {
  const float4 x = __ldg(reinterpret_cast<const float4*>(p));
  r.v[0] = x.x; r.v[1] = x.y; r.v[2] = x.z; r.v[3] = x.w;
}
// Through L2 only: rows that another thread of the same kernel may have written.
__device__ __forceinline__ void row_load_cg(RowVec<8>& r, const float* p) {
  asm volatile("ld.global.cg.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]), "=f"(r.v[4]), "=f"(r.v[5]), "=f"(r.v[6]), "=f"(r.v[7])
               : "l"(p) : "memory");
}
__device__ __forceinline__ void row_load_cg(RowVec<4>& r, const float* p) {
  const float4 x = __ldcg(reinterpret_cast<const float4*>(p));
  r.v[0] = x.x; r.v[1] = x.y; r.v[2] = x.z; r.v[3] = x.w;
}
template <int V> __device__ __forceinline__ void row_zero(RowVec<V>& r) {
#pragma unroll
  for (int e = 0; e < V; ++e) r.v[e] = 0.f;
}
// fp32 store in 16-byte pieces: callers' row buffers are 16-byte aligned, not more.
template <int V> __device__ __forceinline__ void row_store(float* p, const RowVec<V>& r) {
#pragma unroll
  for (int e = 0; e < V; e += 4) *reinterpret_cast<float4*>(p + e) = make_float4(r.v[e], r.v[e + 1], r.v[e + 2], r.v[e + 3]);
}
__device__ __forceinline__ uint32_t row_pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// bf16 store; `wide`: the address is 16-byte aligned (else 8-byte pieces).
__device__ __forceinline__ void row_store_bf16(__nv_bfloat16* p, const RowVec<8>& r, bool wide) {
  const uint4 o = make_uint4(row_pack2(r.v[0], r.v[1]), row_pack2(r.v[2], r.v[3]), row_pack2(r.v[4], r.v[5]), row_pack2(r.v[6], r.v[7]));
  if (wide) {
    *reinterpret_cast<uint4*>(p) = o;
  } else {
    reinterpret_cast<uint2*>(p)[0] = make_uint2(o.x, o.y);
    reinterpret_cast<uint2*>(p)[1] = make_uint2(o.z, o.w);
  }
}
__device__ __forceinline__ void row_store_bf16(__nv_bfloat16* p, const RowVec<4>& r, bool) {
  *reinterpret_cast<uint2*>(p) = make_uint2(row_pack2(r.v[0], r.v[1]), row_pack2(r.v[2], r.v[3]));
}

// Gradients as they lie in memory, converted when they are consumed: all loads of a batch are issued before the first use.
// `wide`: every offset of the batch is a multiple of 8 elements (32 bytes of fp32, 16 bytes of bf16).
template <int V, bool BF16> struct RawVec;
template <> struct RawVec<8, true> {
  uint4 x;
  __device__ __forceinline__ void load(const void* base, long long off, bool wide) {
    const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(base) + off;
    if (wide) {
      x = __ldg(reinterpret_cast<const uint4*>(p));
    } else {
      const uint2 lo = __ldg(reinterpret_cast<const uint2*>(p)), hi = __ldg(reinterpret_cast<const uint2*>(p) + 1);
      x = make_uint4(lo.x, lo.y, hi.x, hi.y);
    }
  }
  __device__ __forceinline__ RowVec<8> get() const {
    RowVec<8> r;
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      r.v[2 * e] = __uint_as_float(w[e] << 16);
      r.v[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
    }
    return r;
  }
};
template <> struct RawVec<4, true> {
  uint2 x;
  __device__ __forceinline__ void load(const void* base, long long off, bool) {
    x = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(base) + off));
  }
  __device__ __forceinline__ RowVec<4> get() const {
    RowVec<4> r;
    r.v[0] = __uint_as_float(x.x << 16); r.v[1] = __uint_as_float(x.x & 0xffff0000u);
    r.v[2] = __uint_as_float(x.y << 16); r.v[3] = __uint_as_float(x.y & 0xffff0000u);
    return r;
  }
};
template <> struct RawVec<8, false> {
  RowVec<8> x;
  __device__ __forceinline__ void load(const void* base, long long off, bool wide) {
    const float* p = reinterpret_cast<const float*>(base) + off;
    if (wide) {
      row_load_nc(x, p);
    } else {
      const float4 lo = __ldg(reinterpret_cast<const float4*>(p)), hi = __ldg(reinterpret_cast<const float4*>(p) + 1);
      x.v[0] = lo.x; x.v[1] = lo.y; x.v[2] = lo.z; x.v[3] = lo.w; x.v[4] = hi.x; x.v[5] = hi.y; x.v[6] = hi.z; x.v[7] = hi.w;
    }
  }
  __device__ __forceinline__ RowVec<8> get() const { return x; }
};
template <> struct RawVec<4, false> {
  RowVec<4> x;
  __device__ __forceinline__ void load(const void* base, long long off, bool) { row_load_nc(x, reinterpret_cast<const float*>(base) + off); }
  __device__ __forceinline__ RowVec<4> get() const { return x; }
};

template <int V> __device__ __forceinline__ void row_atomic_add(float* p, const RowVec<V>& r) {
#pragma unroll
  for (int e = 0; e < V; e += 4) atomicAdd(reinterpret_cast<float4*>(p + e), make_float4(r.v[e], r.v[e + 1], r.v[e + 2], r.v[e + 3]));
}

// peers[r]: the lanes that hold the same key as this one (__match_any_sync).  Leaves in the lowest lane of every such set the
// sum of its v[r].  Equal lanes form a chain in lane order that halves with every step; the R chains step together, and a
// warp without duplicates leaves after one vote.
template <int R>
__device__ __forceinline__ void warp_sum_peers(const unsigned (&peers)[R], float (&v)[R]) {
  const int lane = threadIdx.x & 31;
  int next[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const unsigned above = peers[r] & (0xfffffffeu << lane);
    next[r] = above ? __ffs(above) - 1 : -1;
  }
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    bool done = true;
#pragma unroll
    for (int r = 0; r < R; ++r) done = done && next[r] < 0;
    if (__all_sync(0xffffffffu, done)) break;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int from = next[r] < 0 ? lane : next[r];
      const float o = __shfl_sync(0xffffffffu, v[r], from);
      const int n2 = __shfl_sync(0xffffffffu, next[r], from);
      if (next[r] >= 0) { v[r] += o; next[r] = n2; }
    }
  }
}

// Chooses <V, L, NC> for rows of D floats; `wide`: D is a multiple of 8 and every row starts on a 32-byte boundary.
#define RS_ROW_DISPATCH(wide, D, LAUNCH)                     \
  do {                                                       \
    if (wide) {                                              \
      const int nv_ = (D) / 8;                               \
      if (nv_ <= 4) LAUNCH(8, 4, 1);                         \
      else if (nv_ <= 8) LAUNCH(8, 8, 1);                    \
      else if (nv_ <= 16) LAUNCH(8, 16, 1);                  \
      else if (nv_ <= 32) LAUNCH(8, 32, 1);                  \
      else LAUNCH(8, 32, 2);                                 \
    } else {                                                 \
      const int nv_ = (D) / 4;                               \
      if (nv_ <= 8) LAUNCH(4, 8, 1);                         \
      else if (nv_ <= 32) LAUNCH(4, 32, 1);                  \
      else if (nv_ <= 64) LAUNCH(4, 32, 2);                  \
      else LAUNCH(4, 32, 4);                                 \
    }                                                        \
  } while (0)

inline bool row_wide(const void* weight, int D) { return D % 8 == 0 && (reinterpret_cast<uintptr_t>(weight) & 31) == 0; }

}  // namespace rs
