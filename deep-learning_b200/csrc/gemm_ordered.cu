// Forward products in fp32 with every sum in ascending k, bit for bit what
// gemm_simt.cuh gives, for widths that TMA cannot address and moderate sizes.
//
// What the order is for: a derivative that jumps at 0 (ReLU', the leaky ReLU's, ELU' from
// 1 to 0, SELU') makes a unit's error depend on which side of 0 its pre-activation falls,
// and sums in another order, however accurate, put a few in a million on the other side;
// in a batch of 333 rows one such unit moved the weights after four Adam steps by up to
// 3e-4.  Neither side is the better one.  But these products ran in this order before they
// had another way (as the reference's own loops do), and training on such widths keeps
// giving what it gave where that is cheap (gemm_way in ctx.cu has the line).  Evaluation
// and models without such a derivative take the shortest way that is as accurate.
//
// A CTA forms 64 x 64: four warps of 8 x 4 sums per lane read and multiply, four others
// bring 32 k of both operands at a time, k-major, two slabs ahead (with the loads done by
// the computing warps, through registers, 56 us).  Each lane reads 12 words for 32
// multiply-adds, which bounds a k at 48 shared-memory cycles against 32 of arithmetic;
// with one computing warp to a scheduler it takes 70: 333 x 1203 x 1203 47 us
// (gemm_simt_kernel, 8 words per 16, two barriers per 16 k and no loads under way: 199).
#include <algorithm>

#include "common.cuh"
#include "gemm_store.cuh"
#include "tc_pair.cuh"

namespace dlb {

namespace {

constexpr int OT = 64, OK = 32, O_STAGES = 3;
constexpr int O_COMPUTE = 128, O_THREADS = 256;  // four warps form sums, four load
constexpr int OP = OT + 4;  // pitch of a k-row: 16-byte aligned, banks 4 apart
constexpr int O_TILE = OK * OP;
constexpr int O_LOADS = OT * OK / (O_THREADS - O_COMPUTE);
constexpr int O_SMEM = O_STAGES * 2 * O_TILE * 4;

struct OrderedArgs {
  const float *a, *b;
  long long lda, ldb;
  QuadTarget t;
  int K, tiles_n;
};

// Loader warps: 32 k of 64 lines into a k-major tile, four bytes per copy (a pitch that
// is no multiple of 16 bytes allows no more).  A warp reads 8 k of four lines: whole
// sectors, and stores that touch every bank once.  Beyond the matrix zeros are stored:
// they add nothing.
__device__ __forceinline__ void ordered_load(uint32_t tile, const float *p, long long ld, int line0, int lines, int k0,
                                             int K) {
  const int t = (int)threadIdx.x - O_COMPUTE, lane = t % 32, warp = t / 32;
  const int k = warp * 8 + lane % 8;
  const bool in_k = k0 + k < K;
  const float *src = p + (line0 + lane / 8) * ld + k0 + k;
  const uint32_t dst = tile + (uint32_t)(k * OP + lane / 8) * 4u;
#pragma unroll
  for (int i = 0; i < O_LOADS; ++i) {
    const bool in = in_k && line0 + lane / 8 + 4 * i < lines;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + i * 16u),
                 "l"(in ? src + 4 * i * ld : p), "r"(in ? 4 : 0)
                 : "memory");
  }
}

__global__ void __launch_bounds__(O_THREADS) gemm_ordered_kernel(const __grid_constant__ OrderedArgs g) {
  extern __shared__ __align__(16) float tiles[];  // [stage][A, B][OK][OP]
  pdl_enter();
  const int m0 = (int)blockIdx.x / g.tiles_n * OT, n0 = (int)blockIdx.x % g.tiles_n * OT;
  const int slabs = (g.K + OK - 1) / OK;
  const bool loads = threadIdx.x >= O_COMPUTE;
  const uint32_t base = tc::smem_u32(tiles);
  // A group of copies per slab, empty ones past the end, so that "all but the last
  // group" always means the slab that is read next.
  auto load = [&](int s) {
    if (s < slabs) {
      const uint32_t at = base + (uint32_t)(s % O_STAGES) * 2u * O_TILE * 4u;
      ordered_load(at, g.a, g.lda, m0, g.t.M, s * OK, g.K);
      ordered_load(at + O_TILE * 4u, g.b, g.ldb, n0, g.t.N, s * OK, g.K);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (loads) {
    load(0);
    load(1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
  }
  __syncthreads();
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int mg = warp / 2 % 2 * 32 + lane / 8 * 8, ng = warp % 2 * 32 + lane % 8 * 4;
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int s = 0; s < slabs; ++s) {
    if (loads) {
      load(s + 2);  // its buffer was read in the round before
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      const float *as = tiles + (s % O_STAGES) * 2 * O_TILE + mg, *bs = tiles + (s % O_STAGES) * 2 * O_TILE + O_TILE + ng;
#pragma unroll
      for (int k = 0; k < OK; ++k) {
        const float4 a0 = *reinterpret_cast<const float4 *>(as + k * OP);
        const float4 a1 = *reinterpret_cast<const float4 *>(as + k * OP + 4);
        const float4 b = *reinterpret_cast<const float4 *>(bs + k * OP);
        const float x[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        const float y[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
      }
    }
    __syncthreads();
  }
  if (loads) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    return;
  }
  const float4 b4 = quad_bias(g.t, n0 + ng);
  if (n0 + ng < g.t.N) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (m0 + mg + i < g.t.M) {
        float4 v = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        if (g.t.bias) v.x += b4.x, v.y += b4.y, v.z += b4.z, v.w += b4.w;
        store_quad(g.t, m0 + mg + i, n0 + ng, v);
      }
  }
}

}  // namespace

// About how long it takes.
double gemm_ordered_us(const dlb_ctx *ctx, int M, int N, int K) {
  const long long tiles = (long long)ceil_div(M, OT) * ceil_div(N, OT);
  return 4.0 + 0.036 * K * (double)((tiles + ctx->sm_count - 1) / ctx->sm_count);
}

dlb_status gemm_ordered(dlb_ctx *ctx, const GemmOperand &A, const GemmOperand &B, float *C, long long ldc, int M, int N,
                        int K, const GemmEpilogue &ep) {
  static bool ready[MAX_DEVICES] = {};
  if (!ready[ctx->device]) {
    DLB_CUDA(cudaFuncSetAttribute(gemm_ordered_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, O_SMEM));
    ready[ctx->device] = true;
  }
  const OrderedArgs args{A.ptr, B.ptr, A.stride_mn, B.stride_mn,
                         quad_target(C, ldc, M, N, ep.bias, ep.accumulate, nullptr), K, ceil_div(N, OT)};
  DLB_LAUNCH_KERNEL(ctx, gemm_ordered_kernel, ceil_div(M, OT) * args.tiles_n, O_THREADS, O_SMEM, args);
  DLB_LAUNCHED(ctx);
  ctx->products[DLB_PRODUCT_ORDERED]++;
  return DLB_OK;
}

}  // namespace dlb
