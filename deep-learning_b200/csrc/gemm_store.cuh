// Store of a product's tile from shared memory, four columns of a row per lane: the
// plain store, the store that adds into the output, and the fused epilogues
// (epilogue.cuh) on quads of elements.
//
// The accumulators leave tensor memory with a row per thread; what goes to global
// memory has to be whole rows.  A store that walked the tile row by row, one
// element per lane, took 14000 cycles for 256 x 256 (7 us of a 43 us product at
// 2048^3): one shared-memory load, one bounds check and one store instruction per
// row and 32 columns, each behind the latency of the one before.
#pragma once

#include "common.cuh"
#include "epilogue.cuh"

namespace dlb {

// Where and how the quads of a product go.
struct QuadTarget {
  float *C;
  long long ldc;
  int M, N;
  const float *bias;  // added to every row, or null
  int accumulate;     // C += value
  int atomic;         // C += value from more than one CTA
  int quads;          // rows of C and N allow 16-byte accesses
  const float *col_factor;  // every column times this first (1 / scale of B's lines), or null
};
inline bool quad_aligned(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline QuadTarget quad_target(float *C, long long ldc, int M, int N, const float *bias, int accumulate,
                              const float *col_factor) {
  return QuadTarget{C, ldc, M, N, bias, accumulate, 0, (quad_aligned(C) && (ldc & 3) == 0 && (N & 3) == 0) ? 1 : 0,
                    col_factor};
}

__device__ __forceinline__ float4 quad_of(const float *p, int N, int col, float otherwise) {
  float4 b = make_float4(otherwise, otherwise, otherwise, otherwise);
  if (p) {
    if (col < N) b.x = __ldg(p + col);
    if (col + 1 < N) b.y = __ldg(p + col + 1);
    if (col + 2 < N) b.z = __ldg(p + col + 2);
    if (col + 3 < N) b.w = __ldg(p + col + 3);
  }
  return b;
}
__device__ __forceinline__ float4 quad_bias(const QuadTarget &t, int col) { return quad_of(t.bias, t.N, col, 0.f); }
__device__ __forceinline__ float4 quad_factor(const QuadTarget &t, int col) {
  return quad_of(t.col_factor, t.N, col, 1.f);
}
// v f + b, f a power of two (so that the product is exact).
__device__ __forceinline__ float4 quad_scaled(float4 v, float4 f, float4 b) {
  return make_float4(fmaf(v.x, f.x, b.x), fmaf(v.y, f.y, b.y), fmaf(v.z, f.z, b.z), fmaf(v.w, f.w, b.w));
}

// One quad of a row inside the output, columns col .. col + 3 (col < N).
__device__ __forceinline__ void store_quad(const QuadTarget &t, int row, int col, float4 v) {
  float *dst = t.C + (long long)row * t.ldc + col;
  if (t.quads) {
    if (t.atomic) {
      asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y),
                   "f"(v.z), "f"(v.w)
                   : "memory");
      return;
    }
    if (t.accumulate) {
      const float4 o = *reinterpret_cast<const float4 *>(dst);
      v.x += o.x, v.y += o.y, v.z += o.z, v.w += o.w;
    }
    *reinterpret_cast<float4 *>(dst) = v;
    return;
  }
  const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (col + i < t.N) {
      if (t.atomic) atomicAdd(dst + i, e[i]);
      else dst[i] = t.accumulate ? dst[i] + e[i] : e[i];
    }
}

// f(x) and f'(x, q) of four elements with one dispatch (bit for bit af_fire and
// af_derive).
template <int AF>
__device__ __forceinline__ float4 fire4(float4 x) {
  return make_float4(af_fire(AF, x.x), af_fire(AF, x.y), af_fire(AF, x.z), af_fire(AF, x.w));
}
__device__ __forceinline__ float4 af_fire4(int af, float4 x) {
  switch (af) {
    case DLB_AF_RELU: return fire4<DLB_AF_RELU>(x);
    case DLB_AF_LEAKY_RELU: return fire4<DLB_AF_LEAKY_RELU>(x);
    case DLB_AF_ELU: return fire4<DLB_AF_ELU>(x);
    case DLB_AF_SELU: return fire4<DLB_AF_SELU>(x);
    case DLB_AF_ISRLU: return fire4<DLB_AF_ISRLU>(x);
    default: return x;
  }
}
template <int AF>
__device__ __forceinline__ float4 derive4(float4 x, float4 q) {
  return make_float4(af_derive(AF, x.x, q.x), af_derive(AF, x.y, q.y), af_derive(AF, x.z, q.z),
                     af_derive(AF, x.w, q.w));
}
__device__ __forceinline__ float4 af_derive4(int af, float4 x, float4 q) {
  switch (af) {
    case DLB_AF_RELU: return derive4<DLB_AF_RELU>(x, q);
    case DLB_AF_LEAKY_RELU: return derive4<DLB_AF_LEAKY_RELU>(x, q);
    case DLB_AF_ELU: return derive4<DLB_AF_ELU>(x, q);
    case DLB_AF_SELU: return derive4<DLB_AF_SELU>(x, q);
    case DLB_AF_ISRLU: return derive4<DLB_AF_ISRLU>(x, q);
    default: return make_float4(1.f, 1.f, 1.f, 1.f);
  }
}

// What the fused epilogue reads beside the sums of one quad, loaded ahead of use.
struct FusedLoads {
  float4 a, b;  // EPI_ACTIVATION: a = UOut draws; EPI_DERIVATIVE: a = z, b = activation
};
__device__ __forceinline__ FusedLoads fused_loads(const FusedEpilogue &e, size_t at) {
  FusedLoads l;
  if (e.mode == EPI_DERIVATIVE) {
    l.a = __ldg(reinterpret_cast<const float4 *>(e.z + at));
    l.b = __ldg(reinterpret_cast<const float4 *>(e.a + at));
  } else if (e.noise) {
    l.a = __ldg(reinterpret_cast<const float4 *>(e.noise + at));
  }
  return l;
}

// One quad: `v` = sums + bias.  Stores what the launch asks for (operand planes
// included) and returns the values of the produced operand.  keep: epilogue_keep
// of the four columns.  Element by element the arithmetic of epilogue_store.
__device__ __forceinline__ float4 fused_quad(const FusedEpilogue &e, float *dst, size_t at, float4 v, float4 keep,
                                             const FusedLoads &l, float plane_scale) {
  float4 x;
  if (e.mode == EPI_ACTIVATION) {
    *reinterpret_cast<float4 *>(dst) = v;
    x = af_fire4(e.af, v);
    if (e.noise) {
      x.x = x.x + x.x * l.a.x;
      x.y = x.y + x.y * l.a.y;
      x.z = x.z + x.z * l.a.z;
      x.w = x.w + x.w * l.a.w;
    }
    x.x = keep.x == 0.f ? 0.f : x.x * keep.x;
    x.y = keep.y == 0.f ? 0.f : x.y * keep.y;
    x.z = keep.z == 0.f ? 0.f : x.z * keep.z;
    x.w = keep.w == 0.f ? 0.f : x.w * keep.w;
    *reinterpret_cast<float4 *>(e.out + at) = x;
  } else {
    const float4 d = af_derive4(e.af, l.a, l.b);
    x = make_float4(v.x * d.x, v.y * d.y, v.z * d.z, v.w * d.w);
    *reinterpret_cast<float4 *>(dst) = x;
  }
  if (e.sink.hi) {
    const float p[4] = {x.x, x.y, x.z, x.w};
    sink_store4(e.sink, at, p, plane_scale);
  }
  return x;
}

// Range statistics of the quads a lane stores, all of the same four columns.  The
// `lanes` (a power of two) lanes of a row are neighbours.
struct QuadTracker {
  unsigned cm[4] = {0u, 0u, 0u, 0u};
  __device__ __forceinline__ void row(const PlaneSink &k, int r, bool live, float4 x, int lanes) {
    const unsigned b0 = live ? abs_bits(x.x) : 0u, b1 = live ? abs_bits(x.y) : 0u, b2 = live ? abs_bits(x.z) : 0u,
                   b3 = live ? abs_bits(x.w) : 0u;
    cm[0] = max(cm[0], b0), cm[1] = max(cm[1], b1), cm[2] = max(cm[2], b2), cm[3] = max(cm[3], b3);
    if (k.rowmax) {  // every lane of the warp is here
      unsigned m = max(max(b0, b1), max(b2, b3));
      for (int o = lanes >> 1; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      if ((threadIdx.x & (unsigned)(lanes - 1)) == 0 && m) atomicMax(k.rowmax + r, m);
    }
  }
  // Lanes `lanes` apart hold the same columns.
  __device__ __forceinline__ void finish(const PlaneSink &k, int col, int n, int lanes) {
    for (int o = lanes; o < 32; o <<= 1)
#pragma unroll
      for (int j = 0; j < 4; ++j) cm[j] = max(cm[j], __shfl_xor_sync(0xffffffffu, cm[j], o));
    if (k.colmax && (int)(threadIdx.x & 31u) < lanes && col < n) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (cm[j]) atomicMax(k.colmax + col + j, cm[j]);
    }
    if (k.slot) {
      const unsigned all = max(max(cm[0], cm[1]), max(cm[2], cm[3]));
      amax_commit(reinterpret_cast<unsigned *>(k.slot) + SLOT_AMAX, all);
    }
  }
};

}  // namespace dlb
