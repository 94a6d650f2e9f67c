// Products of a few million multiply-adds, on the CUDA cores in fp32.
//
// Such a product is all latency: the tensor-core kernels take 8 - 12 us for 128 x 784 x
// 256 (set-up of tensor memory and barriers, conversion of the operands, drain), of
// which the arithmetic would be a tenth, and their operand planes cost launches of
// their own.  Here a CTA forms a 32 x 32 tile over a part of k: 128 k of both operands
// at a time go through registers into shared memory, k-major, the next 128 under way
// while these are used; each of the eight warps takes 16 of the 128 k and the whole
// tile, 8 x 4 sums per lane, so that a value read from shared memory is used four
// or eight times; the warps' tiles are added through shared memory.  Where the tiles
// leave SMs idle up to eight CTAs (a cluster) share a tile's k range and add through
// each other's shared memory.  Any stride and size; 12 shared-memory cycles per k and
// warp and the stores into shared memory bound a chunk (1.5 us), launch and latency the
// rest: 128 x 784 x 256 11.7 -> 6.0 us, 1 x 784 x 256 10.2 -> 4.6, 256^3 10.5 -> 5.4.
#include <algorithm>

#include "common.cuh"
#include "gemm_store.cuh"
#include "tc_pair.cuh"

namespace dlb {

namespace {

constexpr int ST = 32;           // rows and columns of a tile
constexpr int SK = 128;          // k per chunk
constexpr int S_THREADS = 256;
constexpr int S_WARPS = S_THREADS / 32;
constexpr int SP = ST + 4;       // pitch of a k-row: 16-byte aligned, banks 4 apart
constexpr int S_LOADS = ST * SK / S_THREADS;
constexpr int S_MAX_SHIFT = 3;

struct SmallArgs {
  const float *a, *b;
  long long a_mn, a_k, b_mn, b_k;
  QuadTarget t;
  int K, tiles_n, split_shift;
};

// This thread's 16 elements of lines [line0, line0 + 32) x k [k0, k0 + 128).  k
// contiguous: a warp reads 8 k of four lines (whole 32-byte sectors, and the store into
// k-rows 36 words apart touches every bank once); otherwise 32 lines of one k.
template <bool MN>
__device__ __forceinline__ void place(int i, int *line, int *k) {
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  if (MN) {
    *line = lane;
    *k = i * S_WARPS + warp;
  } else {
    *line = warp * 4 + lane / 8;
    *k = i * 8 + lane % 8;
  }
}
template <bool MN>
__device__ __forceinline__ void fetch(float (&v)[S_LOADS], const float *p, long long s_mn, long long s_k, int line0,
                                      int lines, int k0, int k1) {
#pragma unroll
  for (int i = 0; i < S_LOADS; ++i) {
    int line, k;
    place<MN>(i, &line, &k);
    line += line0, k += k0;
    v[i] = line < lines && k < k1 ? __ldg(p + line * s_mn + k * s_k) : 0.f;
  }
}
template <bool MN>
__device__ __forceinline__ void put(float *tile, const float (&v)[S_LOADS]) {
#pragma unroll
  for (int i = 0; i < S_LOADS; ++i) {
    int line, k;
    place<MN>(i, &line, &k);
    tile[k * SP + line] = v[i];
  }
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(S_THREADS, 2) gemm_small_kernel(const __grid_constant__ SmallArgs g) {
  __shared__ __align__(16) float tiles[2 * SK * SP];
  static_assert(2 * SK * SP >= S_WARPS * ST * SP, "the warps' tiles fit where the operands were");
  pdl_enter();
  const int splits = 1 << g.split_shift;
  const int rank = (int)blockIdx.x & (splits - 1), tile_id = (int)blockIdx.x >> g.split_shift;
  const int m0 = tile_id / g.tiles_n * ST, n0 = tile_id % g.tiles_n * ST;
  const int k_begin = (int)((long long)g.K * rank >> g.split_shift), k_end = (int)((long long)g.K * (rank + 1) >> g.split_shift);
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32, mg = lane / 8 * 8, ng = lane % 8 * 4;
  float *as = tiles, *bs = tiles + SK * SP;
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  float va[S_LOADS], vb[S_LOADS];
  fetch<A_MN>(va, g.a, g.a_mn, g.a_k, m0, g.t.M, k_begin, k_end);
  fetch<B_MN>(vb, g.b, g.b_mn, g.b_k, n0, g.t.N, k_begin, k_end);
  for (int k0 = k_begin; k0 < k_end; k0 += SK) {
    put<A_MN>(as, va);
    put<B_MN>(bs, vb);
    __syncthreads();
    if (k0 + SK < k_end) {
      fetch<A_MN>(va, g.a, g.a_mn, g.a_k, m0, g.t.M, k0 + SK, k_end);
      fetch<B_MN>(vb, g.b, g.b_mn, g.b_k, n0, g.t.N, k0 + SK, k_end);
    }
    // Warp w takes k = w, w + 8, ...: short ends of a k range fall to all of them.
    const int used = min(SK, k_end - k0);
#pragma unroll 4
    for (int k = warp; k < used; k += S_WARPS) {
      const float4 a0 = *reinterpret_cast<const float4 *>(as + k * SP + mg);
      const float4 a1 = *reinterpret_cast<const float4 *>(as + k * SP + mg + 4);
      const float4 b = *reinterpret_cast<const float4 *>(bs + k * SP + ng);
      const float x[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float y[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
    }
    __syncthreads();
  }
  // The eight warps' tiles, then the CTAs'.
#pragma unroll
  for (int i = 0; i < 8; ++i)
    *reinterpret_cast<float4 *>(tiles + (warp * ST + mg + i) * SP + ng) =
        make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  __syncthreads();
  const int row = threadIdx.x / 8, col = threadIdx.x % 8 * 4;
  float *const at = tiles + row * SP + col;
  float4 v = *reinterpret_cast<const float4 *>(at);
#pragma unroll
  for (int w = 1; w < S_WARPS; ++w) {
    const float4 u = *reinterpret_cast<const float4 *>(at + w * ST * SP);
    v.x += u.x, v.y += u.y, v.z += u.z, v.w += u.w;
  }
  bool mine = true;
  if (splits > 1) {
    *reinterpret_cast<float4 *>(at) = v;  // its own place in the first warp's tile
    tc::cluster_sync_all();
    mine = (row << g.split_shift) / ST == rank;
    if (mine) {
      v = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int r = 0; r < splits; ++r) {
        float4 u;
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(u.x), "=f"(u.y), "=f"(u.z), "=f"(u.w)
                     : "r"(tc::map_to_cta(tc::smem_u32(at), (uint32_t)r)));
        v.x += u.x, v.y += u.y, v.z += u.z, v.w += u.w;
      }
    }
  }
  if (mine && m0 + row < g.t.M && n0 + col < g.t.N) {
    const float4 b4 = quad_bias(g.t, n0 + col);
    store_quad(g.t, m0 + row, n0 + col, make_float4(v.x + b4.x, v.y + b4.y, v.z + b4.z, v.w + b4.w));
  }
  if (splits > 1) tc::cluster_sync_all();  // no CTA leaves while another reads its sums
}

int small_tiles(int M, int N) { return ceil_div(M, ST) * ceil_div(N, ST); }

// CTAs that share a tile's k range: as long as that fills idle SMs and leaves 32 k each.
int small_split_shift(const dlb_ctx *ctx, int M, int N, int K) {
  const long long tiles = (long long)ceil_div(M, ST) * ceil_div(N, ST);
  int shift = 0;
  while (shift < S_MAX_SHIFT && (tiles << (shift + 1)) <= ctx->sm_count && (K >> (shift + 1)) >= 32) ++shift;
  return shift;
}

template <bool A_MN, bool B_MN>
dlb_status launch_small(dlb_ctx *ctx, const SmallArgs &args, int tiles) {
  DLB_CUDA(launch_kernel_cluster(ctx, gemm_small_kernel<A_MN, B_MN>, dim3((unsigned)(tiles << args.split_shift)),
                                 dim3(S_THREADS), 0, 1u << args.split_shift, args));
  DLB_LAUNCHED(ctx);
  ctx->products[DLB_PRODUCT_SMALL]++;
  return DLB_OK;
}

}  // namespace

// About how long it takes: 1.6 us a chunk, and more where an SM has several CTAs (512^3,
// two to an SM: 15.8 us; 300 x 1024 x 300, three: 15.6).
double gemm_small_us(const dlb_ctx *ctx, int M, int N, int K) {
  const int shift = small_split_shift(ctx, M, N, K);
  const long long ctas = ((long long)ceil_div(M, ST) * ceil_div(N, ST)) << shift;
  const int chunks = ceil_div(ceil_div(K, 1 << shift), SK);
  const double per_sm = (double)((ctas + ctx->sm_count - 1) / ctx->sm_count);
  return 3.2 + (shift ? 0.8 : 0.0) + chunks * std::max(1.6, 1.45 * per_sm);
}

dlb_status gemm_small(dlb_ctx *ctx, const GemmOperand &A, const GemmOperand &B, float *C, long long ldc, int M, int N,
                      int K, const GemmEpilogue &ep) {
  const SmallArgs args{A.ptr, B.ptr, A.stride_mn, A.stride_k, B.stride_mn, B.stride_k,
                       quad_target(C, ldc, M, N, ep.bias, ep.accumulate, nullptr), K, ceil_div(N, ST),
                       small_split_shift(ctx, M, N, K)};
  const bool a_mn = A.stride_k != 1, b_mn = B.stride_k != 1;
  const int tiles = small_tiles(M, N);
  if (a_mn) return b_mn ? launch_small<true, true>(ctx, args, tiles) : launch_small<true, false>(ctx, args, tiles);
  return b_mn ? launch_small<false, true>(ctx, args, tiles) : launch_small<false, false>(ctx, args, tiles);
}

}  // namespace dlb
