// Noise of the step drawn on the device: Bernoulli dropout masks, UOut draws
// and ShakeDrop flags and factors, as an alternative to the arrays that the
// host hands over (the reference draws them from per-thread generators during
// the step: Model::Dropout_Bernoulli, Forward_Pass__Dropout__Uout__OpenMP
// fwp_mp.cpp L:4959-4985, Forward_Pass__Dropout__ShakeDrop__OpenMP L:4922-4957;
// those streams depend on the thread count and cannot be reproduced, so only
// the distributions are the reference's).
//
// The generator is Philox4x32-10 (Salmon, Moraes, Dror, Shaw: "Parallel random
// numbers: as easy as 1, 2, 3", SC'11): a keyed bijection of a 128-bit counter,
// ten rounds of two 32x32->64 multiplications.  Element i of a draw is word
// i mod 4 of the block with counter (i / 4, stream, step) and key = seed, so a
// draw is a pure function of (seed, stream, step, first + i): ranks that hold
// different rows of a batch draw their slices of the same array, and the union
// does not depend on how the rows are sharded.
#include "common.cuh"

namespace dlb {

namespace {

constexpr uint32_t PHILOX_M0 = 0xD2511F53u, PHILOX_M1 = 0xCD9E8D57u;
constexpr uint32_t PHILOX_W0 = 0x9E3779B9u, PHILOX_W1 = 0xBB67AE85u;

__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
#pragma unroll
  for (int round = 0; round < 10; ++round) {
    const uint32_t hi0 = __umulhi(PHILOX_M0, c.x), lo0 = PHILOX_M0 * c.x;
    const uint32_t hi1 = __umulhi(PHILOX_M1, c.z), lo1 = PHILOX_M1 * c.z;
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    k.x += PHILOX_W0;
    k.y += PHILOX_W1;
  }
  return c;
}

// 24 random bits -> [0, 1).
__device__ __forceinline__ float unit_float(uint32_t x) { return (float)(x >> 8) * (1.f / 16777216.f); }

struct NoiseKey {
  uint2 key;        // seed
  uint32_t stream;  // which array of the step
  uint32_t step;
  uint64_t first;   // index of out[0] in the whole array
};

__device__ __forceinline__ uint4 block_of(const NoiseKey &k, uint64_t block) {
  return philox4x32_10(make_uint4((uint32_t)block, (uint32_t)(block >> 32), k.stream, k.step), k.key);
}

__device__ __forceinline__ uint32_t word_of(const uint4 &v, int w) {
  return w == 0 ? v.x : (w == 1 ? v.y : (w == 2 ? v.z : v.w));
}

// One thread per generator block (four consecutive elements of the array).
template <typename Emit>
__device__ __forceinline__ void for_each_word(const NoiseKey &k, size_t n, Emit emit) {
  const uint64_t first_block = k.first / 4, last_block = (k.first + n + 3) / 4;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = first_block + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < last_block; b += stride) {
    const uint4 v = block_of(k, b);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const uint64_t i = b * 4 + w;
      if (i >= k.first && i < k.first + n) emit((size_t)(i - k.first), word_of(v, w));
    }
  }
}

__global__ void __launch_bounds__(256) uniform_kernel(float *__restrict__ out, size_t n, float lo, float width, NoiseKey k) {
  pdl_enter();
  // Two roundings (no fused multiply-add), so that a host restatement in fp32
  // gives the same bits.
  for_each_word(k, n, [=](size_t i, uint32_t x) { out[i] = __fadd_rn(__fmul_rn(unit_float(x), width), lo); });
}

__global__ void __launch_bounds__(256) bernoulli_kernel(uint8_t *__restrict__ out, size_t n, float p, NoiseKey k) {
  pdl_enter();
  for_each_word(k, n, [=](size_t i, uint32_t x) { out[i] = unit_float(x) < p ? 1 : 0; });
}

// ShakeDrop's flags, and the forward and backward factors of the flagged rows: what the
// three draws give, without the rows nobody reads (at a probability that grows to 1/2
// over the layers, three quarters of two arrays of 8 MB).  One warp per row; VEC: whole
// generator blocks of a row.  2048 x 1024: three launches of 11.8 us together -> one of 5.6.
template <bool VEC>
__global__ void __launch_bounds__(256)
    shakedrop_kernel(uint8_t *__restrict__ mask, float *__restrict__ fwd, float *__restrict__ bwd, size_t rows,
                     size_t width, float p, NoiseKey km, NoiseKey kf, NoiseKey kb) {
  pdl_enter();
  const int lane = threadIdx.x % 32;
  const size_t warps = (size_t)gridDim.x * (blockDim.x / 32);
  for (size_t r = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; r < rows; r += warps) {
    const uint64_t at = km.first + r;
    const bool flag = unit_float(word_of(block_of(km, at / 4), (int)(at % 4))) < p;
    if (lane == 0) mask[r] = flag ? 1 : 0;
    if (!flag) continue;
    const size_t row = r * width;
    if (VEC) {
      for (size_t c = (size_t)lane * 4; c < width; c += 128) {
        const uint4 f = block_of(kf, (kf.first + row + c) / 4), b = block_of(kb, (kb.first + row + c) / 4);
        auto forward = [](uint32_t x) { return __fadd_rn(__fmul_rn(unit_float(x), 2.f), -1.f); };
        *reinterpret_cast<float4 *>(fwd + row + c) = make_float4(forward(f.x), forward(f.y), forward(f.z), forward(f.w));
        *reinterpret_cast<float4 *>(bwd + row + c) =
            make_float4(unit_float(b.x), unit_float(b.y), unit_float(b.z), unit_float(b.w));
      }
    } else {
      for (size_t c = lane; c < width; c += 32) {
        const uint64_t i = kf.first + row + c;
        const int w = (int)(i % 4);
        fwd[row + c] = __fadd_rn(__fmul_rn(unit_float(word_of(block_of(kf, i / 4), w)), 2.f), -1.f);
        bwd[row + c] = unit_float(word_of(block_of(kb, i / 4), w));
      }
    }
  }
}

NoiseKey make_key(uint64_t seed, uint32_t stream, uint32_t step, uint64_t first) {
  NoiseKey k;
  k.key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
  k.stream = stream;
  k.step = step;
  k.first = first;
  return k;
}

int noise_blocks(dlb_ctx *ctx, size_t n) {
  return (int)std::max<size_t>(1, std::min<size_t>((n / 4 + 256) / 256, (size_t)ctx->sm_count * 16));
}

}  // namespace

}  // namespace dlb

using namespace dlb;

dlb_status dlb::noise_shakedrop(dlb_ctx *ctx, uint8_t *mask, float *fwd, float *bwd, size_t rows, size_t width, float p,
                                uint64_t seed, uint32_t stream, uint32_t step, uint64_t first_row) {
  DLB_REQUIRE(ctx && mask && fwd && bwd && rows > 0 && width > 0 && p >= 0.f && p <= 1.f, "noise_shakedrop");
  const NoiseKey km = make_key(seed, stream, step, first_row), kf = make_key(seed, stream + 1, step, first_row * width),
                 kb = make_key(seed, stream + 2, step, first_row * width);
  const int grid = (int)std::min<size_t>((rows + 7) / 8, (size_t)ctx->sm_count * 16);
  const bool vec = width % 4 == 0 && ((reinterpret_cast<uintptr_t>(fwd) | reinterpret_cast<uintptr_t>(bwd)) & 15) == 0;
  if (vec) DLB_LAUNCH_KERNEL(ctx, shakedrop_kernel<true>, grid, 256, 0, mask, fwd, bwd, rows, width, p, km, kf, kb);
  else DLB_LAUNCH_KERNEL(ctx, shakedrop_kernel<false>, grid, 256, 0, mask, fwd, bwd, rows, width, p, km, kf, kb);
  DLB_LAUNCHED(ctx);
  return DLB_OK;
}

extern "C" {

dlb_status dlb_noise_uniform(dlb_ctx *ctx, float *out, size_t n, float lo, float hi, uint64_t seed,
                             uint32_t stream, uint32_t step, uint64_t first) {
  DLB_REQUIRE(ctx && (out || n == 0) && hi >= lo, "dlb_noise_uniform");
  if (n == 0) return DLB_OK;
  DLB_LAUNCH_KERNEL(ctx, uniform_kernel, noise_blocks(ctx, n), 256, 0, out, n, lo, hi - lo, make_key(seed, stream, step, first));
  DLB_LAUNCHED(ctx);
  return DLB_OK;
}

dlb_status dlb_noise_bernoulli(dlb_ctx *ctx, uint8_t *out, size_t n, float p, uint64_t seed, uint32_t stream,
                               uint32_t step, uint64_t first) {
  DLB_REQUIRE(ctx && (out || n == 0) && p >= 0.f && p <= 1.f, "dlb_noise_bernoulli");
  if (n == 0) return DLB_OK;
  DLB_LAUNCH_KERNEL(ctx, bernoulli_kernel, noise_blocks(ctx, n), 256, 0, out, n, p, make_key(seed, stream, step, first));
  DLB_LAUNCHED(ctx);
  return DLB_OK;
}

}  // extern "C"
