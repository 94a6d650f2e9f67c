// FC product straight from the fp32 tensors: C[m,n] (+)= sum_k A(m,k) B(n,k) for
// operands of any size, pitch and alignment, without plane buffers.
//
// The plane kernels (gemm_pair.cu, gemm_tcgen05.cu) read operands that were
// split into fp16 planes beforehand and that TMA can address, and gemm_small.cu takes
// a few million multiply-adds; what lies between (outputs below a 256 x 256 tile
// with a long k, outputs for which making planes first takes longer) ran on the CUDA
// cores, one 64 x 64 tile per block whatever K.  Here sixteen warps read fp32, split it in
// registers and write the swizzled operand tiles the tensor core reads:
//
//   converters  warps 0-15   8 lines of A and 8 of B per chunk of 64 k each, the
//                            next 8 lines in flight while these convert; in turn
//                            they issue a chunk's MMAs, three products
//                            lo hi + hi lo + hi hi per 16 k
//   drain       warps 16-31  add each finished chunk into fp32 registers, 32 columns
//                            each
//
// Scale.  Every line (row of A, row of B^T) of every chunk has a power-of-two
// scale of its own, s max|x| in [2^14, 2^15) over the line's 64 values; the
// drain multiplies a chunk by both inverse scales, exactly.  Every value of a
// line that is within 2^-17 of the largest of its 64 neighbours has the full
// 22 bits whatever the rest of the tensor looks like, so there is no range
// guard here: nothing to flag.  A line with a value of 2^101 or more, infinity or
// NaN sends its tile through the fp32 body at the end instead.
//
// Accumulation.  A chunk is 64 deep: two accumulator buffers of 128 columns in
// tensor memory, each drained with round-to-nearest adds, so the tensor core's
// truncating adder only sees sums of 64 products.
//
// What bounds it: the conversion.  A chunk of a 128 x 128 tile takes about 5000 cycles
// where its MMAs take 768: 12000 instructions of loads, line maxima, splits and
// stores, and their latencies.  That is why larger outputs go to the plane kernels,
// whose operands are split once: 333 x 1203 x 1203 takes 25 us here (172 us on the CUDA
// cores), 1024 x 1000 x 2048 54 (6 + 17 on planes).  A small output has few tiles: up to eight CTAs of a cluster
// then share a tile's k range, and each adds the others' parts of its slice of
// columns through distributed shared memory, in rank order, so that results
// do not depend on timing.
#include "common.cuh"
#include "gemm_simt.cuh"
#include "tc_pair.cuh"

namespace dlb {

namespace {

using namespace tc;

constexpr int DM = 128, DN = 128;   // tile
constexpr int DK = 64;              // depth of a chunk: one 128-byte row of halfs
constexpr int D_STAGES = 2;         // operand tiles in shared memory, with their line scales and accumulators
constexpr int D_CONV_WARPS = 16;
constexpr int D_DRAIN_WARPS = 16;
constexpr int D_LINES = DM / D_CONV_WARPS;       // lines of an operand per converter warp and chunk
constexpr int D_COLS = DN / (D_DRAIN_WARPS / 4); // accumulator columns per drain warp
constexpr int D_THREADS = 32 * (D_CONV_WARPS + D_DRAIN_WARPS);
constexpr int D_PLANE = DM * DK * 2;             // one plane of one operand, 16 KB
constexpr int D_STAGE = 4 * D_PLANE;             // A hi, A lo, B hi, B lo
constexpr int D_PARTS = D_STAGES * D_STAGE;      // partial sums of this CTA's columns, from every CTA of the cluster
constexpr int D_PART_BYTES = DM * (DN + 8 * 4) * 4;
constexpr int D_SCALES = D_PARTS + D_PART_BYTES; // [D_STAGES][DM + DN] floats
constexpr int D_BARS = D_SCALES + D_STAGES * (DM + DN) * 4;
constexpr int D_MAX_SHIFT = 3;
constexpr int D_SMEM = D_BARS + 128 + 1024;
static_assert(D_COLS == 32 && D_LINES == 8, "fragment sizes below");
static_assert(D_SMEM <= 232448, "shared memory of one CTA");

struct DirectArgs {
  SimtOperands o;
  float *C;
  long long ldc;
  int M, N, K;
  const float *bias;
  int accumulate;
  int tiles_n;
  int split_shift;   // log2 of the CTAs of a cluster, each with its share of the chunks
  int *status;
};

__device__ __forceinline__ void sts128(uint32_t addr, const uint32_t (&v)[4]) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
               : "memory");
}
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}

// Packed fp32 pairs: one instruction for two multiplications or additions.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// Two values to their halves: the roundings of plane_halves (x s is exact, so
// x s - hi in one fused operation is too).
__device__ __forceinline__ void split2(float a, float b, uint64_t s, uint32_t *hi, uint32_t *lo) {
  const uint64_t x = pack2(a, b);
  const float2 t = unpack2(mul2(x, s));
  const __half2 h = __floats2half2_rn(t.x, t.y);
  const float2 f = __half22float2(__hneg2(h));
  const float2 d = unpack2(fma2(x, s, pack2(f.x, f.y)));
  const __half2 l = __floats2half2_rn(d.x, d.y);
  *hi = *reinterpret_cast<const uint32_t *>(&h);
  *lo = *reinterpret_cast<const uint32_t *>(&l);
}

// The 8 lines of one operand that a converter warp owns in a chunk, 16 values per
// lane:
//   MN = false (k contiguous): eight lanes to a line, two lines each.  The lanes of
//     quarter w = lane / 8 hold of line row_line(step, w) the values 4 (lane & 7) ..
//     + 3 and 32 further on, step 0 in r[0..7] and step 1 in r[8..15].
//   MN = true (mn contiguous): line lane & 7, its values 16 (lane / 8) + i in r[i].
// Both read whole 32-byte sectors.  Lines and k outside the operand read as zero.
// The order of the lines puts rows r and r + 4 of the tile into one half of the
// warp, whose 8-byte stores then cover all banks under the swizzle.
__device__ __forceinline__ int row_line(int step, int lane) { return 2 * step + (lane >> 4) + 4 * ((lane >> 3) & 1); }

// Whether base and pitch allow 16-byte loads along a line.
__device__ __forceinline__ bool quads_aligned(const float *x, long long pitch) {
  return (((unsigned)(reinterpret_cast<uintptr_t>(x) >> 2) | (unsigned)pitch) & 3u) == 0;
}

template <bool MN>
__device__ __forceinline__ void load_lines(float (&r)[16], const float *__restrict__ x, long long pitch, int mn0,
                                           int mn_end, int k0, int k_end, bool quads, int lane) {
  if (MN) {
    const int mn = mn0 + (lane & 7), k = k0 + (lane >> 3) * 16;
    const float *p = x + (long long)k * pitch + mn;
    const int n = mn < mn_end ? k_end - k : 0;  // values of this lane inside the operand
    if (n >= 16) {
#pragma unroll
      for (int i = 0; i < 16; ++i) r[i] = __ldg(p + i * pitch);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) r[i] = i < n ? __ldg(p + i * pitch) : 0.f;
    }
  } else {
    const int k = k0 + 4 * (lane & 7);
#pragma unroll
    for (int step = 0; step < 2; ++step) {
      const int mn = mn0 + row_line(step, lane);
      const float *p = x + (long long)mn * pitch + k;
      float *t = r + 8 * step;
      if (quads && mn0 + D_LINES <= mn_end && k0 + DK <= k_end) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float4 v = __ldg(reinterpret_cast<const float4 *>(p + 32 * i));
          t[4 * i] = v.x, t[4 * i + 1] = v.y, t[4 * i + 2] = v.z, t[4 * i + 3] = v.w;
        }
      } else {
        const int n = mn < mn_end ? k_end - k : 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int at = (i & 3) + 32 * (i >> 2);
          t[i] = at < n ? __ldg(p + at) : 0.f;
        }
      }
    }
  }
}

// s = 2^(14 - E) for a line whose largest |x| has exponent E, the scale of
// plane_scale_from_bits(bits, PLANE_EXP_OWN) as integer arithmetic on the biased
// exponent, and 1 / s.  Exponents below -112 count as -112: s stays below 2^127.
__device__ __forceinline__ unsigned line_scale_bits(unsigned max_bits) {
  const unsigned e = max(max_bits, 15u << 23) & 0x7f800000u;
  return ((unsigned)(2 * 127 + PLANE_EXP_OWN) << 23) - e;
}
__device__ __forceinline__ float line_inverse(unsigned scale_bits) {
  return __uint_as_float((254u << 23) - scale_bits);
}

// Splits the lines and writes them as rows `row0 ..` (a multiple of 8) of a k-major
// tile under the 128-byte swizzle (16-byte piece c of row r lies at piece
// c ^ (r & 7)); the inverse scales go to inv[row0 ..].  Returns whether a value is
// out of range.
template <bool MN>
__device__ __forceinline__ bool convert_lines(const float (&r)[16], uint32_t hi, uint32_t lo, float *inv, int row0,
                                              int lane) {
  constexpr float TOO_LARGE = 2.5353012e30f;  // 2^101
  if (MN) {
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) m = fmaxf(m, fabsf(r[i]));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
    const unsigned sb = line_scale_bits(__float_as_uint(m));
    const uint64_t s = pack2(__uint_as_float(sb), __uint_as_float(sb));
    const int line = lane & 7;
    if (lane < 8) inv[row0 + line] = line_inverse(sb);
    const uint32_t row = (uint32_t)((row0 + line) * 128);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t h[4], l[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) split2(r[8 * c + 2 * j], r[8 * c + 2 * j + 1], s, &h[j], &l[j]);
      const uint32_t at = row + (uint32_t)((((lane >> 3) * 2 + c) ^ line) << 4);
      sts128(hi + at, h);
      sts128(lo + at, l);
    }
    return m >= TOO_LARGE;
  } else {
    bool large = false;
#pragma unroll
    for (int step = 0; step < 2; ++step) {
      const float *t = r + 8 * step;
      float m = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(t[i]));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
      large |= m >= TOO_LARGE;
      const unsigned sb = line_scale_bits(__float_as_uint(m));
      const uint64_t s = pack2(__uint_as_float(sb), __uint_as_float(sb));
      const int line = row_line(step, lane);
      if ((lane & 7) == 0) inv[row0 + line] = line_inverse(sb);
      const uint32_t at = (uint32_t)((row0 + line) * 128 + ((((lane & 7) >> 1) ^ line) << 4) + (lane & 1) * 8);
      uint32_t h[4], l[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) split2(t[2 * j], t[2 * j + 1], s, &h[j], &l[j]);
      sts64(hi + at, h[0], h[1]);
      sts64(hi + (at ^ 64u), h[2], h[3]);
      sts64(lo + at, l[0], l[1]);
      sts64(lo + (at ^ 64u), l[2], l[3]);
    }
    return large;
  }
}

// A tile with a value outside what the halves can hold: its 64 x 64 quarters in
// fp32, shared out among the CTAs of the cluster.  A call of its own, so that its
// registers are not part of the kernel's main path.
__device__ __noinline__ void direct_fp32_tile(const DirectArgs *a, int m0, int n0, int piece, float *shared) {
  const int tn = (a->N + ST_N - 1) / ST_N;
  for (int i = piece; i < 4; i += 1 << a->split_shift) {
    const int m = m0 + (i >> 1) * ST_M, n = n0 + (i & 1) * ST_N;
    if (m < a->M && n < a->N)
      gemm_simt_body(a->o, a->C, a->ldc, a->M, a->N, a->K, a->bias, a->accumulate, shared, (m / ST_M) * tn + n / ST_N,
                     0x40000000);
  }
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(D_THREADS, 1) gemm_direct_kernel(const __grid_constant__ DirectArgs a) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (base - raw);
  float *scales = reinterpret_cast<float *>(smem + D_SCALES);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + D_BARS);
  // full: the converters have written a chunk; done: its MMAs are complete;
  // empty: it has been drained; parts: the cluster's partial sums are here.
  const uint32_t full0 = smem_u32(bars), done0 = full0 + 8 * D_STAGES, empty0 = done0 + 8 * D_STAGES,
                 parts_bar = empty0 + 8 * D_STAGES;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 3 * D_STAGES + 1);
  int *range_flag = reinterpret_cast<int *>(bars + 3 * D_STAGES + 1) + 1;
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(range_flag + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int splits = 1 << a.split_shift;
  if (threadIdx.x == 0) {
    for (int s = 0; s < D_STAGES; ++s) {
      mbar_init(full0 + 8 * s, D_CONV_WARPS);
      mbar_init(done0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, D_DRAIN_WARPS);
    }
    mbar_init(parts_bar, (uint32_t)(D_DRAIN_WARPS * splits));
    *abort_flag = 0;
    *range_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == D_CONV_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                 "r"((uint32_t)(D_STAGES * DN))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = *tmem_holder;
  // The cluster's other CTAs may write here from now on; the wait for theirs comes
  // before the first remote access.
  if (splits > 1) cluster_arrive();
  // The set-up above touches no global memory: it runs under the kernel before.
  pdl_enter();

  const int piece = (int)(blockIdx.x & (unsigned)(splits - 1)), tile_id = (int)(blockIdx.x >> a.split_shift);
  const int m0 = (tile_id / a.tiles_n) * DM, n0 = (tile_id % a.tiles_n) * DN;
  const int total = (a.K + DK - 1) / DK;
  const int c_begin = (int)(((long long)piece * total) >> a.split_shift);
  const int chunks = (int)(((long long)(piece + 1) * total) >> a.split_shift) - c_begin;
  const int cols = min(DN, a.N - n0);
  const int n_mma = (cols + 15) & ~15;  // columns the MMAs form

  float acc[D_COLS];
  const int q = warp & 3, g = (warp - D_CONV_WARPS) >> 2;
  int s = 0;
  uint32_t phase = 0;
  if (warp < D_CONV_WARPS) {
    // ---------------- converters ----------------
    const int line0 = warp * D_LINES;
    const bool do_a = m0 + line0 < a.M, do_b = n0 + line0 < a.N;
    const long long a_pitch = A_MN ? a.o.a_sk : a.o.a_sm, b_pitch = B_MN ? a.o.b_sk : a.o.b_sn;
    const bool a_quads = quads_aligned(a.o.A, a_pitch), b_quads = quads_aligned(a.o.B, b_pitch);
    const uint32_t idesc = (1u << 4) | ((uint32_t)(n_mma >> 3) << 17) | ((uint32_t)(DM >> 4) << 24);
    float ra[16], rb[16];
    bool bad = false;
    int k0 = c_begin * DK;
    if (do_a) load_lines<A_MN>(ra, a.o.A, a_pitch, m0 + line0, a.M, k0, a.K, a_quads, lane);
    for (int c = 0; c < chunks; ++c, k0 += DK) {
      if (do_b) load_lines<B_MN>(rb, a.o.B, b_pitch, n0 + line0, a.N, k0, a.K, b_quads, lane);
      if (!__all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, phase ^ 1, abort_flag, a.status))) break;
      const uint32_t st = base + s * D_STAGE;
      float *inv = scales + s * (DM + DN);
      if (do_a) bad |= convert_lines<A_MN>(ra, st, st + D_PLANE, inv, line0, lane);
      if (do_a && c + 1 < chunks) load_lines<A_MN>(ra, a.o.A, a_pitch, m0 + line0, a.M, k0 + DK, a.K, a_quads, lane);
      if (do_b) bad |= convert_lines<B_MN>(rb, st + 2 * D_PLANE, st + 3 * D_PLANE, inv + DM, line0, lane);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(full0 + 8 * s);
        // The MMAs of chunk c are warp (c mod 16)'s to issue.
        if ((c & (D_CONV_WARPS - 1)) == warp && mbar_wait(full0 + 8 * s, phase, abort_flag, a.status)) {
          tcgen05_fence_after();
          const uint32_t d = tmem + (uint32_t)(s * DN);
          // (a step of 16 k is 32 bytes: 2 in the descriptors' address field)
          const uint64_t a_hi = make_smem_desc(st, 16, 1024, LAYOUT_SW128),
                         a_lo = make_smem_desc(st + D_PLANE, 16, 1024, LAYOUT_SW128),
                         b_hi = make_smem_desc(st + 2 * D_PLANE, 16, 1024, LAYOUT_SW128),
                         b_lo = make_smem_desc(st + 3 * D_PLANE, 16, 1024, LAYOUT_SW128);
#pragma unroll
          for (int k = 0; k < DK / 16; ++k) {
            umma_f16(d, a_lo + 2 * k, b_hi + 2 * k, idesc, k ? 1u : 0u);
            umma_f16(d, a_hi + 2 * k, b_lo + 2 * k, idesc, 1u);
            umma_f16(d, a_hi + 2 * k, b_hi + 2 * k, idesc, 1u);
          }
          umma_commit(done0 + 8 * s);
        }
      }
      __syncwarp();
      if (++s == D_STAGES) s = 0, phase ^= 1;
    }
    if (bad) *range_flag = 1;
  } else {
    // ---------------- drain ----------------
#pragma unroll
    for (int j = 0; j < D_COLS; ++j) acc[j] = 0.f;
    const bool live = g * D_COLS < n_mma;
    for (int c = 0; c < chunks; ++c) {
      if (!__all_sync(0xffffffffu, mbar_wait(done0 + 8 * s, phase, abort_flag, a.status))) break;
      if (live) {
        tcgen05_fence_after();
        const float *inv = scales + s * (DM + DN);
        const float fa = inv[q * 32 + lane];
        const uint64_t fa2 = pack2(fa, fa);
        uint32_t v[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(s * DN + g * D_COLS), v);
#pragma unroll
        for (int i = 0; i < D_COLS; i += 4) {
          const ulonglong2 fb = *reinterpret_cast<const ulonglong2 *>(inv + DM + g * D_COLS + i);
          const float2 x = unpack2(fma2(mul2(pack2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), fb.x), fa2,
                                        pack2(acc[i], acc[i + 1])));
          const float2 y = unpack2(fma2(mul2(pack2(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])), fb.y), fa2,
                                        pack2(acc[i + 2], acc[i + 3])));
          acc[i] = x.x, acc[i + 1] = x.y, acc[i + 2] = y.x, acc[i + 3] = y.y;
        }
        tcgen05_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty0 + 8 * s);
      if (++s == D_STAGES) s = 0, phase ^= 1;
    }
  }

  // ---------------- sum of the pieces, store ----------------
  // CTA r of the cluster owns columns [r width, (r + 1) width) of the tile and is
  // sent every CTA's part of them, one arrival per drain warp; rows are padded by
  // four words so that the 16-byte stores of a warp's 32 rows spread over the banks.
  const int width_shift = 7 - a.split_shift, width = 1 << width_shift, row_words = width + 4;
  tcgen05_fence_before();
  __syncthreads();  // the range flag is final
  if (splits > 1) cluster_wait();
  if (warp >= D_CONV_WARPS) {
    if (g * D_COLS < n_mma) {
      const int row = q * 32 + lane;
#pragma unroll
      for (int j = 0; j < D_COLS; j += 4) {
        const int col = g * D_COLS + j, owner = col >> width_shift;
        const uint32_t at = base + D_PARTS + (uint32_t)(((piece * DM + row) * row_words + col - (owner << width_shift)) * 4);
        st_cluster4(splits > 1 ? map_to_cta(at, (uint32_t)owner) : at, acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
      }
    }
    if (splits > 1) {
      const int bad = *reinterpret_cast<volatile int *>(range_flag);
      if (bad && lane < splits) st_cluster_int(map_to_cta(smem_u32(range_flag), (uint32_t)lane), 1);
      asm volatile("fence.acq_rel.cluster;" ::: "memory");
      __syncwarp();
      if (lane < splits) mbar_arrive_cluster(map_to_cta(parts_bar, (uint32_t)lane));
    } else {
      __syncwarp();
      if (lane == 0) mbar_arrive(parts_bar);
    }
  }
  // Everything this thread sends is on its way.  The CTAs leave together (at the end):
  // one whose own wait ran out must not be gone while another still writes its part here.
  __syncwarp();
  if (splits > 1) cluster_arrive();
  const bool here = mbar_wait_cluster(parts_bar, 0, abort_flag, a.status);
  if (*reinterpret_cast<volatile int *>(range_flag)) {
    direct_fp32_tile(&a, m0, n0, piece, reinterpret_cast<float *>(smem));
  } else if (here) {
    const float *part = reinterpret_cast<const float *>(smem + D_PARTS);
    const int own0 = n0 + (piece << width_shift), own_cols = min(width, a.N - own0), rows = min(DM, a.M - m0);
    const int stride = DM * row_words, tx = threadIdx.x & (width - 1);  // lanes run along a row
    if (tx < own_cols) {
      const float b = a.bias ? __ldg(a.bias + own0 + tx) : 0.f;
      for (int r = threadIdx.x >> width_shift; r < rows; r += D_THREADS >> width_shift) {
        const float *src = part + r * row_words + tx;
        float v = src[0];
        for (int p = 1; p < splits; ++p) v += src[p * stride];
        v += b;
        float *dst = a.C + (long long)(m0 + r) * a.ldc + own0 + tx;
        *dst = a.accumulate ? *dst + v : v;
      }
    }
  }
  __syncwarp();
  if (splits > 1) cluster_wait();
  if (*abort_flag) drain_pause();  // MMAs that were issued
  if (warp == D_CONV_WARPS) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)(D_STAGES * DN))
                 : "memory");
  }
}

int clusters_at_once(const dlb_ctx *ctx, int shift) {
  static int known[MAX_DEVICES][D_MAX_SHIFT + 1] = {};
  int &n = known[ctx->device][shift];
  if (n == 0) n = resident_clusters(ctx, gemm_direct_kernel<false, false>, D_THREADS, D_SMEM, 1 << shift);
  return n;
}

// CTAs per tile: as many as the chip runs at once (16 tiles by clusters of eight are
// two rounds on 148 SMs: 512^3 22 us against 14), each with a chunk at least.
int direct_split_shift(const dlb_ctx *ctx, int M, int N, int K) {
  const int tiles = ceil_div(M, DM) * ceil_div(N, DN), chunks = ceil_div(K, DK);
  int s = 0;
  while (s < D_MAX_SHIFT && tiles <= clusters_at_once(ctx, s + 1) && (2 << s) <= chunks) ++s;
  return s;
}

template <bool A_MN, bool B_MN>
dlb_status launch_direct(dlb_ctx *ctx, const DirectArgs &args, int tiles) {
  auto kernel = gemm_direct_kernel<A_MN, B_MN>;
  static bool attr_set[MAX_DEVICES] = {};
  if (!attr_set[ctx->device]) {
    DLB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, D_SMEM));
    attr_set[ctx->device] = true;
  }
  DLB_CUDA(launch_kernel_cluster(ctx, kernel, dim3((unsigned)(tiles << args.split_shift)), dim3(D_THREADS), D_SMEM,
                                 1u << args.split_shift, args));
  DLB_LAUNCHED(ctx);
  ctx->products[DLB_PRODUCT_DIRECT]++;
  return DLB_OK;
}

}  // namespace

dlb_status gemm_direct(dlb_ctx *ctx, const GemmOperand &A, const GemmOperand &B, float *C, long long ldc, int M, int N,
                       int K, const GemmEpilogue &ep) {
  DirectArgs args{SimtOperands{A.ptr, A.stride_mn, A.stride_k, B.ptr, B.stride_mn, B.stride_k}, C, ldc, M, N, K,
                  ep.bias, ep.accumulate, ceil_div(N, DN), direct_split_shift(ctx, M, N, K), ctx->d_status};
  const int tiles = args.tiles_n * ceil_div(M, DM);
  const bool a_mn = A.stride_k != 1, b_mn = B.stride_k != 1;
  if (a_mn) return b_mn ? launch_direct<true, true>(ctx, args, tiles) : launch_direct<true, false>(ctx, args, tiles);
  return b_mn ? launch_direct<false, true>(ctx, args, tiles) : launch_direct<false, false>(ctx, args, tiles);
}

double gemm_direct_us(const dlb_ctx *ctx, int M, int N, int K) {
  const int shift = direct_split_shift(ctx, M, N, K);
  const long long ctas = (long long)ceil_div(M, DM) * ceil_div(N, DN) << shift;
  const long long rounds = (ctas + ctx->sm_count - 1) / ctx->sm_count;
  return 7.5 + 3.0 * (double)rounds * ceil_div(ceil_div(K, DK), 1 << shift);
}

bool gemm_direct_supported(const GemmOperand &A, const GemmOperand &B) {
  return (A.stride_k == 1 || A.stride_mn == 1) && (B.stride_k == 1 || B.stride_mn == 1);
}

}  // namespace dlb
