// The fp16-plane FC product for outputs of a few hundred to a few thousand rows and
// columns: C[m,n] (+)= sum_k A(m,k) B(n,k).
//
// gemm_x3_pair_kernel gives 256 x 256 tiles to pairs of SMs; 1024 x 1024 outputs are
// 16 tiles for 74 pairs, and a product of any size lasts as long as one whole
// tile.  Here a pair's tile is 256 x 128 and up to four pairs of a cluster share a
// tile's k range, so that such an output fills the chip.  One tile per cluster, not
// persistent.
//
// A k-block is 64 deep (128-byte rows).  With blocks of 32 the one thread that
// issues the MMAs needed 660 - 760 cycles per block whatever the tile's width
// (waits, commits, descriptors), as much as the tensor cores need for 256 columns;
// a block of 64 costs it about the same, for twice the work.
//
// Roles per CTA: warp 0 loads with TMA, warp 1 issues the MMAs (in the even CTA of
// a pair), warps 2-9 drain the accumulator chunks into registers; all ten warps
// store.  Barriers of a pair as in gemm_x3_pair_kernel.
//
// Sum of the pieces.  At the end every CTA holds 128 rows x 128 columns of partial
// sums.  It lays them out in its own, now idle, operand ring, in one block per
// owner: of the S CTAs of a cluster with the same rows, CTA p owns columns
// [128 p / S, 128 (p + 1) / S).  One bulk copy per owner takes a block to the owner's
// receive buffer (distributed shared memory; thread stores to remote memory, 16
// bytes of each of 32 rows per instruction, moved 8 bytes per clock, bulk copies
// 17 - 31), and the owner adds the parts in order of k, so that results do not
// depend on timing.  16-byte slot c of a row r lies at c ^ (r & 7): rows are written by
// thread, read by lane.
//
// An MN-major operand is fetched in boxes of 64 lines {64 mn, 64 k}: unlike the
// 3-d view of the pair kernel's maps, this asks nothing of the extent but a
// pitch of whole 16-byte units.  Chunks are two k-blocks (128 deep), half of the
// pair kernel's, for a smaller share of truncated sums: 4.8e-7 against 9.3e-7 of
// the float64 product.
//
// A store leaves an SM at 32 bytes per clock (measured, any pattern of whole
// lines), so the 64 KB of a CTA's tile part take 2050 cycles whatever the kernel does.
#include <stdlib.h>

#include "common.cuh"
#include "gemm_simt.cuh"
#include "gemm_store.cuh"
#include "tc_pair.cuh"

namespace dlb {

namespace {

using namespace tc;

constexpr int QM = 256, QN = 128;  // a pair's tile
constexpr int QK = 64;             // halfs per k-block (128-byte rows)
constexpr int Q_CHUNK = 2;         // k-blocks per accumulator drain
constexpr int Q_STAGES = 3;
constexpr int Q_A = BM * QK * 2;        // this CTA's 128 rows of A, one plane
constexpr int Q_B = (QN / 2) * QK * 2;  // this CTA's 64 columns of B, one plane
constexpr int Q_STAGE = 2 * Q_A + 2 * Q_B;
constexpr int Q_RING = Q_STAGES * Q_STAGE;
constexpr int Q_TILE_BYTES = BM * QN * 4;                 // this CTA's part of the tile
constexpr int Q_MAX_SHIFT = 2;                            // four pieces
constexpr int Q_RECEIVE = Q_RING;                         // the other pieces' blocks
constexpr int Q_RECEIVE_BYTES = Q_TILE_BYTES * 3 / 4;     // S - 1 blocks of 1 / S of a tile part
constexpr int Q_BARS = Q_RECEIVE + Q_RECEIVE_BYTES;
constexpr int Q_SMEM = Q_BARS + 256 + 1024;
static_assert(Q_RING >= Q_TILE_BYTES, "the ring holds the tile part");
static_assert(Q_SMEM <= 232448, "shared memory of one CTA");

struct MidArgs {
  QuadTarget t;
  int K, tiles_n;
  const float *scale_a, *scale_b, *line_inv_a;
  const unsigned *guard_a, *guard_b;
  unsigned mask_a, mask_b;
  SimtOperands fp32;
  unsigned long long *fallbacks;
  int *status;
};

// LINES lines of one plane.
template <bool MN, int LINES>
__device__ __forceinline__ void load_plane(uint32_t dst, const CUtensorMap *map, uint32_t bar, int line0, int k0) {
  if (MN) {
#pragma unroll
    for (int g = 0; g < LINES / 64; ++g) tma_pair_2d(dst + g * 64 * QK * 2, map, bar, line0 + g * 64, k0);
  } else {
    tma_pair_2d(dst, map, bar, k0, line0);
  }
}

// This CTA's block for another one, into that one's receive buffer.
__device__ __forceinline__ void send_block(uint32_t dst_cluster, uint32_t src, uint32_t bytes, uint32_t bar_cluster) {
  asm volatile(
      "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_cluster),
      "r"(src), "r"(bytes), "r"(bar_cluster)
      : "memory");
}

template <bool A_MN, bool B_MN, bool FUSED, int SHIFT>
__global__ void __launch_bounds__(NUM_THREADS, 1)
    gemm_mid_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_a_lo,
                    const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_b_lo,
                    const __grid_constant__ MidArgs a, const __grid_constant__ FusedEpilogue fe) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (base - raw);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + Q_BARS);
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * Q_STAGES, acc_full0 = empty0 + 8 * Q_STAGES,
                 acc_empty0 = acc_full0 + 16, parts_bar = acc_empty0 + 16;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 2 * Q_STAGES + 5);
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bars + 2 * Q_STAGES + 6);
  unsigned *issued_kb = reinterpret_cast<unsigned *>(bars + 2 * Q_STAGES + 7);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  constexpr int SPLITS = 1 << SHIFT;  // pairs that share the tile
  const uint32_t rank = cluster_rank(), half = rank & 1u, lead = rank & ~1u;
  const int piece = (int)(rank >> 1);
  if (threadIdx.x == 0) {
    for (int s = 0; s < Q_STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);   // the even CTA's producer; bytes of both CTAs' loads
      mbar_init(empty0 + 8 * s, 1);  // one commit
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full0 + 8 * b, 1);
      mbar_init(acc_empty0 + 8 * b, 2 * NUM_DRAIN_WARPS);  // drain warps of both CTAs
    }
    mbar_init(parts_bar, 1);
    if (SPLITS > 1) mbar_expect_tx(parts_bar, (uint32_t)(Q_TILE_BYTES - (Q_TILE_BYTES >> SHIFT)));
    *abort_flag = 0;
    *issued_kb = 0;
    prefetch_tmap(&tm_a);
    prefetch_tmap(&tm_a_lo);
    prefetch_tmap(&tm_b);
    prefetch_tmap(&tm_b_lo);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                 "r"((uint32_t)(2 * QN))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();  // every CTA's barriers exist before anything arrives on them
  tcgen05_fence_after();
  const uint32_t tmem = *tmem_holder;
  // The set-up above touches no global memory: it runs under the kernel before.
  pdl_enter();

  const int tile_id = (int)(blockIdx.x >> (SHIFT + 1));
  const int m0 = (tile_id / a.tiles_n) * QM + (int)half * BM, n0 = (tile_id % a.tiles_n) * QN;
  const int total_kb = (a.K + QK - 1) / QK;
  const int kb_begin = (int)(((long long)piece * total_kb) >> SHIFT);
  const int num_kb = (int)(((long long)(piece + 1) * total_kb) >> SHIFT) - kb_begin;
  // Range guard: the planes may not stand for an operand.  The words arrive while
  // the first k-blocks do; a flagged product is computed again below.
  const bool flagged = (a.guard_a && (*a.guard_a & a.mask_a)) || (a.guard_b && (*a.guard_b & a.mask_b));

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      const uint32_t lead_full0 = map_to_cta(full0, lead);
      const int b0 = n0 + (int)half * (QN / 2);
      for (int kb = 0; kb < num_kb; ++kb) {
        const int s = kb % Q_STAGES;
        if (!mbar_wait(empty0 + 8 * s, ((kb / Q_STAGES) & 1) ^ 1, abort_flag, a.status)) break;
        const uint32_t fb = lead_full0 + 8 * s, st = base + s * Q_STAGE;
        if (half == 0) mbar_expect_tx(full0 + 8 * s, 2 * Q_STAGE);
        const int k0 = (kb_begin + kb) * QK;
        load_plane<A_MN, BM>(st, &tm_a, fb, m0, k0);
        load_plane<A_MN, BM>(st + Q_A, &tm_a_lo, fb, m0, k0);
        load_plane<B_MN, QN / 2>(st + 2 * Q_A, &tm_b, fb, b0, k0);
        load_plane<B_MN, QN / 2>(st + 2 * Q_A + Q_B, &tm_b_lo, fb, b0, k0);
        *issued_kb = (unsigned)kb + 1;
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (even CTA of the pair) ----------------
    if (lane == 0 && half == 0) {
      const uint32_t idesc = (1u << 4) | ((A_MN ? 1u : 0u) << 15) | ((B_MN ? 1u : 0u) << 16) |
                             ((uint32_t)(QN >> 3) << 17) | ((uint32_t)(QM >> 4) << 24);
      // Swizzled 128-byte rows for either major; steps in the descriptors' address
      // field are 16 bytes.
      constexpr uint32_t A_LBO = A_MN ? QK * 128 : 16, B_LBO = B_MN ? QK * 128 : 16;
      constexpr uint32_t A_STEP = (A_MN ? 16 * 128 : 32) >> 4, B_STEP = (B_MN ? 16 * 128 : 32) >> 4;
      const uint64_t desc_a = make_smem_desc(base, A_LBO, 1024, LAYOUT_SW128),
                     desc_b = make_smem_desc(base + 2 * Q_A, B_LBO, 1024, LAYOUT_SW128);
      bool ok = true;
      int s = 0;
      uint32_t phase = 0;
      for (int kb = 0, cc = 0; kb < num_kb && ok; ++cc) {
        const int buf = cc & 1;
        ok = mbar_wait(acc_empty0 + 8 * buf, ((cc >> 1) & 1) ^ 1, abort_flag, a.status);
        if (!ok) break;
        tcgen05_fence_after();
        const uint32_t d = tmem + (uint32_t)(buf * QN);
        const int kb_end = min(num_kb, kb + Q_CHUNK);
        uint32_t add = 0u;
        for (; kb < kb_end; ++kb) {
          ok = mbar_wait(full0 + 8 * s, phase, abort_flag, a.status);
          if (!ok) break;
          tcgen05_fence_after();
          const uint64_t a_hi = desc_a + (uint64_t)(s * (Q_STAGE >> 4)), b_hi = desc_b + (uint64_t)(s * (Q_STAGE >> 4));
#pragma unroll
          for (int k = 0; k < QK / 16; ++k) {
            umma_pair_f16(d, a_hi + (Q_A >> 4) + k * A_STEP, b_hi + k * B_STEP, idesc, add);
            umma_pair_f16(d, a_hi + k * A_STEP, b_hi + (Q_B >> 4) + k * B_STEP, idesc, 1u);
            umma_pair_f16(d, a_hi + k * A_STEP, b_hi + k * B_STEP, idesc, 1u);
            add = 1u;
          }
          umma_pair_commit(empty0 + 8 * s, lead);
          if (++s == Q_STAGES) s = 0, phase ^= 1;
        }
        if (ok) umma_pair_commit(acc_full0 + 8 * buf, lead);
      }
    }
  } else {
    // ---------------- drain: warps 2..9 of every CTA ----------------
    const int q = warp & 3, h = (warp - 2) >> 2;
    const float out_b = a.t.col_factor ? 1.f : 1.f / __ldg(a.scale_b);
    const int row = q * 32 + lane;
    const float out_a = a.line_inv_a ? __ldg(a.line_inv_a + min(m0 + row, a.t.M - 1)) : 1.f / __ldg(a.scale_a);
    const uint32_t lead_acc_empty0 = map_to_cta(acc_empty0, lead);
    float acc[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) acc[j] = 0.f;
    const int chunks = (num_kb + Q_CHUNK - 1) / Q_CHUNK;
    for (int c = 0; c < chunks; ++c) {
      const int buf = c & 1;
      const bool ok = mbar_wait(acc_full0 + 8 * buf, (c >> 1) & 1, abort_flag, a.status);
      if (!__all_sync(0xffffffffu, ok)) break;
      tcgen05_fence_after();
      const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * QN + h * 64);
#pragma unroll
      for (int j = 0; j < 64; j += 32) {
        uint32_t v[32];
        tmem_ld32(taddr + j, v);
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[j + i] += __uint_as_float(v[i]);
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(lead_acc_empty0 + 8 * buf);
    }
    // The last chunk is complete, so no MMA or load of this pair touches the ring any
    // more.  (out_a is this row's factor, so scaling here scales every part alike.)
    constexpr int width_shift = 7 - SHIFT;
    float4 *stage = reinterpret_cast<float4 *>(smem);
#pragma unroll
    for (int j = 0; j < 64; j += 4) {
      const int col = h * 64 + j, owner = col >> width_shift, slot = (col - (owner << width_shift)) >> 2;
      stage[(((owner * BM + row) << width_shift) >> 2) + (slot ^ (row & 7))] =
          make_float4(acc[j] * out_a * out_b, acc[j + 1] * out_a * out_b, acc[j + 2] * out_a * out_b,
                      acc[j + 3] * out_a * out_b);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();

  if (flagged) {
    // fp32 on the CUDA cores, every CTA taking its share of the 64 x 64 tiles; every
    // CTA reads the same words.
    if (a.fallbacks && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(a.fallbacks, 1ull);
    gemm_simt_guard_path(a.fp32, a.t.C, a.t.ldc, a.t.M, a.t.N, a.K, a.t.bias, a.t.accumulate,
                         reinterpret_cast<float *>(smem), FUSED ? &fe : nullptr);
  } else {
    // ---------------- sum of the pieces and store, all warps ----------------
    constexpr int width_shift = 7 - SHIFT;
    constexpr int block_bytes = Q_TILE_BYTES >> SHIFT;
    if (SPLITS > 1 && threadIdx.x < SPLITS && (int)threadIdx.x != piece && *abort_flag == 0) {
      // To piece p: its block of this CTA's part, into the slot for this piece.
      const int p = threadIdx.x;
      const uint32_t to = (uint32_t)(2 * p) + half, slot = (uint32_t)(piece < p ? piece : piece - 1);
      send_block(map_to_cta(base + Q_RECEIVE + slot * block_bytes, to), base + (uint32_t)(p * block_bytes),
                 (uint32_t)block_bytes, map_to_cta(parts_bar, to));
    }
    constexpr int WARPS = NUM_THREADS / 32;
    constexpr int quads_shift = width_shift - 2;   // quads, and lanes, of a row: 32, 16 or 8
    constexpr int lanes = 1 << quads_shift;
    // Warp w takes units w, w + 10, ... of 32 quads each; a lane keeps its columns.
    const int quad0 = (warp * 32 + lane) & ((1 << quads_shift) - 1);
    const int col = n0 + (piece << width_shift) + quad0 * 4;
    const float4 b4 = quad_bias(a.t, col), f4 = quad_factor(a.t, col);
    const bool live = col < a.t.N;
    const bool plain = !FUSED && a.t.quads && !a.t.accumulate;
    const float plane_scale = FUSED && fe.sink.hi ? sink_scale(fe.sink) : 1.f;
    float4 keep = b4;
    if (FUSED && live)
      keep = make_float4(epilogue_keep(fe, col), epilogue_keep(fe, col + 1), epilogue_keep(fe, col + 2),
                         epilogue_keep(fe, col + 3));
    bool here = true;
    if (SPLITS > 1) here = mbar_wait_cluster(parts_bar, 0, abort_flag, a.status);
    if (here) {
      const float4 *own = reinterpret_cast<const float4 *>(smem) + ((piece * BM) << quads_shift);
      const float4 *others = reinterpret_cast<const float4 *>(smem + Q_RECEIVE);
      constexpr int units = (BM << quads_shift) / 32;
      QuadTracker track;
      constexpr int AHEAD = 4;
#pragma unroll 1
      for (int u = warp; u < units; u += AHEAD * WARPS) {
        FusedLoads in[AHEAD];
        float4 v[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
          const int r = ((u + i * WARPS) * 32 + lane) >> quads_shift;
          if (FUSED && live && r < BM && m0 + r < a.t.M) in[i] = fused_loads(fe, (size_t)(m0 + r) * a.t.N + col);
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
          const int r = ((u + i * WARPS) * 32 + lane) >> quads_shift;
          if (r < BM) {
            const int at = (r << quads_shift) + (quad0 ^ (r & 7));
            if (SPLITS == 1) {
              v[i] = own[at];
            } else {
              v[i] = piece == 0 ? own[at] : others[at];
#pragma unroll
              for (int p = 1; p < SPLITS; ++p) {
                const float4 w = p == piece ? own[at] : others[((p < piece ? p : p - 1) * (BM << quads_shift)) + at];
                v[i].x += w.x, v[i].y += w.y, v[i].z += w.z, v[i].w += w.w;
              }
            }
            v[i] = quad_scaled(v[i], f4, b4);
          }
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
          const int r = ((u + i * WARPS) * 32 + lane) >> quads_shift, row = m0 + r;
          const bool inside = live && r < BM && row < a.t.M;
          if (plain) {
            if (inside) *reinterpret_cast<float4 *>(a.t.C + (long long)row * a.t.ldc + col) = v[i];
          } else if (!FUSED) {
            if (inside) store_quad(a.t, row, col, v[i]);
          } else {
            const size_t at = (size_t)row * a.t.N + col;
            if (inside) v[i] = fused_quad(fe, a.t.C + at, at, v[i], keep, in[i], plane_scale);
            track.row(fe.sink, row, inside, v[i], lanes);
          }
        }
      }
      if (FUSED) track.finish(fe.sink, col, a.t.N, lanes);
    }
  }

  // ---------------- teardown ----------------
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0 && half == 0) {
    const unsigned issued = *issued_kb;
    const long long t0 = clock64();
    for (unsigned kb = issued > (unsigned)Q_STAGES ? issued - Q_STAGES : 0; kb < issued; ++kb) {
      while (!mbar_try_wait(full0 + 8 * (kb % Q_STAGES), (kb / Q_STAGES) & 1)) {
        if (clock64() - t0 > DRAIN_BUDGET_CLOCKS) break;
      }
    }
  }
  __syncthreads();
  cluster_sync_all();  // no CTA leaves while another may still signal it or write its parts
  if (*abort_flag) drain_pause();  // blocks sent to this CTA that it did not wait for
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)(2 * QN))
                 : "memory");
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace {

template <bool A_MN, bool B_MN, bool FUSED, int SHIFT>
dlb_status launch_mid_shift(dlb_ctx *ctx, const GemmOperand &A, const GemmOperand &B, float *C, long long ldc, int M, int N,
                      int K, const GemmEpilogue &ep) {
  CUtensorMap ta, tal, tb, tbl;
  const bool ok = tmap_plane(ctx, &ta, A_MN, A.h_hi, M, K, A_MN ? A.stride_k : A.stride_mn, QK, BM) &&
                  tmap_plane(ctx, &tal, A_MN, A.h_lo, M, K, A_MN ? A.stride_k : A.stride_mn, QK, BM) &&
                  tmap_plane(ctx, &tb, B_MN, B.h_hi, N, K, B_MN ? B.stride_k : B.stride_mn, QK, QN / 2) &&
                  tmap_plane(ctx, &tbl, B_MN, B.h_lo, N, K, B_MN ? B.stride_k : B.stride_mn, QK, QN / 2);
  if (!ok) {
    set_error("gemm_mid: cuTensorMapEncodeTiled rejected an operand");
    return DLB_ERR_CUDA;
  }
  auto kernel = gemm_mid_kernel<A_MN, B_MN, FUSED, SHIFT>;
  static bool attr_set[MAX_DEVICES] = {};
  if (!attr_set[ctx->device]) {
    DLB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Q_SMEM));
    attr_set[ctx->device] = true;
  }
  const int tiles_n = ceil_div(N, QN), tiles = tiles_n * ceil_div(M, QM);
  const MidArgs args{quad_target(C, ldc, M, N, ep.bias, ep.accumulate, B.line_inv), K, tiles_n, A.scale, B.scale,
                     A.line_inv, A.guard, B.guard, A.guard_mask, B.guard_mask,
                     fp32_operands(A, B),
                     ctx->d_guard ? ctx->d_guard + 1 : nullptr, ctx->d_status};
  DLB_CUDA(launch_kernel_cluster(ctx, kernel, dim3((unsigned)(tiles << (SHIFT + 1))), dim3(NUM_THREADS), Q_SMEM,
                                 2u << SHIFT, ta, tal, tb, tbl, args, FUSED ? *ep.fused : FusedEpilogue{}));
  DLB_LAUNCHED(ctx);
  ctx->products[DLB_PRODUCT_MID]++;
  return DLB_OK;
}

template <bool A_MN, bool B_MN, bool FUSED>
dlb_status launch_mid(dlb_ctx *ctx, const GemmOperand &A, const GemmOperand &B, float *C, long long ldc, int M, int N,
                      int K, int split_shift, const GemmEpilogue &ep) {
  switch (split_shift) {
    case 0: return launch_mid_shift<A_MN, B_MN, FUSED, 0>(ctx, A, B, C, ldc, M, N, K, ep);
    case 1: return launch_mid_shift<A_MN, B_MN, FUSED, 1>(ctx, A, B, C, ldc, M, N, K, ep);
    default: return launch_mid_shift<A_MN, B_MN, FUSED, 2>(ctx, A, B, C, ldc, M, N, K, ep);
  }
}

int clusters_at_once(const dlb_ctx *ctx, int shift) {
  static int known[MAX_DEVICES][Q_MAX_SHIFT + 1] = {};
  int &n = known[ctx->device][shift];
  if (n == 0)
    n = resident_clusters(ctx,
                          shift == 0   ? gemm_mid_kernel<false, false, false, 0>
                          : shift == 1 ? gemm_mid_kernel<false, false, false, 1>
                                       : gemm_mid_kernel<false, false, false, 2>,
                          NUM_THREADS, Q_SMEM, 2 << shift);
  return n;
}

}  // namespace

dlb_status gemm_mid(dlb_ctx *ctx, const GemmOperand &A, const GemmOperand &B, float *C, long long ldc, int M, int N,
                    int K, int split_shift, const GemmEpilogue &ep) {
  const bool a_mn = !(A.stride_k == 1), b_mn = !(B.stride_k == 1);
  if (ep.fused && ep.fused->mode != EPI_PLAIN) {
    if (!a_mn && !ep.accumulate)
      return b_mn ? launch_mid<false, true, true>(ctx, A, B, C, ldc, M, N, K, split_shift, ep)
                  : launch_mid<false, false, true>(ctx, A, B, C, ldc, M, N, K, split_shift, ep);
    set_error("gemm_mid: no fused epilogue for this layout");
    return DLB_ERR_UNSUPPORTED;
  }
  if (!a_mn && !b_mn) return launch_mid<false, false, false>(ctx, A, B, C, ldc, M, N, K, split_shift, ep);
  if (!a_mn && b_mn) return launch_mid<false, true, false>(ctx, A, B, C, ldc, M, N, K, split_shift, ep);
  if (a_mn && b_mn) return launch_mid<true, true, false>(ctx, A, B, C, ldc, M, N, K, split_shift, ep);
  set_error("gemm_mid: MN-major A with K-major B is not instantiated");
  return DLB_ERR_UNSUPPORTED;
}

// The number of pieces of the k range that makes the product shortest, as a shift,
// and about how long it then takes.
double gemm_mid_us(const dlb_ctx *ctx, int M, int N, int K, int *split_shift) {
  const long long tiles = (long long)ceil_div(M, QM) * ceil_div(N, QN);
  const int kb = ceil_div(K, QK);
  double best = 1e30;
  for (int s = 0; s <= Q_MAX_SHIFT; ++s) {
    if (s && kb < (Q_CHUNK << s)) break;  // a chunk at least per piece
    const int at_once = clusters_at_once(ctx, s);
    const long long rounds = (tiles + at_once - 1) / at_once;
    const double us = 2.5 + (double)rounds * (4.5 + (s ? 0.8 : 0.0) + 0.55 * ceil_div(kb, 1 << s));
    if (us < best) {
      best = us;
      *split_shift = s;
    }
  }
  return best;
}

}  // namespace dlb
