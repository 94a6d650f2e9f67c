// Operand planes of the tensor-core products.
//
// 3xFP16: a tensor x is used as hi + lo with hi = fp16(s x), lo = fp16(s x - hi),
// s a power of two per tensor chosen from max |x| so that s max lies in
// [2^14, 2^15).  The plane buffer of a tensor (its `_lo` argument in the C ABI)
// has the tensor's byte size and holds the hi plane followed by the lo plane.
// The context remembers, under the buffer's address, which tensor was split
// into it, its element count and the device slot of s; the FC entry points
// look their `_lo` arguments up there.
#include <cuda_fp16.h>
#include <string.h>

#include "common.cuh"
#include "planes.cuh"
#include "tc_pair.cuh"

namespace dlb {

namespace {

// Largest |x| as raw bits (monotonic for non-negative floats).
__global__ void absmax_kernel(const float *__restrict__ x, size_t n, unsigned *slot) {
  pdl_enter();
  unsigned m = 0;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t n4 = n / 4;
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  if (vec) {
#pragma unroll 4
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(x) + i);
      m = max(max(m, v.x & 0x7fffffffu), max(v.y & 0x7fffffffu, max(v.z & 0x7fffffffu, v.w & 0x7fffffffu)));
    }
    for (size_t i = n4 * 4 + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
      m = max(m, __float_as_uint(x[i]) & 0x7fffffffu);
  } else {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
      m = max(m, __float_as_uint(x[i]) & 0x7fffffffu);
  }
  for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (threadIdx.x % 32 == 0 && m > *reinterpret_cast<volatile unsigned *>(slot)) atomicMax(slot, m);
}

// Flat split of a tensor without a shape (or one whose rows are not a whole
// number of float4): planes only, no line statistics.
__global__ void split_flat_kernel(const float *__restrict__ x, size_t n, PlaneSink k) {
  pdl_enter();
  const float s = sink_scale(k);
  __half *hi = reinterpret_cast<__half *>(k.hi), *lo = reinterpret_cast<__half *>(k.lo);
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const bool vec = ((reinterpret_cast<uintptr_t>(x) & 15) | (reinterpret_cast<uintptr_t>(hi) & 7) |
                    (reinterpret_cast<uintptr_t>(lo) & 7)) == 0;
  const size_t n4 = vec ? n / 4 : 0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(x) + i);
    const float a[4] = {v.x, v.y, v.z, v.w};
    sink_store4(k, i * 4, a, s);
  }
  for (size_t i = n4 * 4 + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    plane_halves(x[i], s, hi + i, lo + i);
}

// Split of a [rows, cols] tensor (cols a multiple of 4) with the row and column
// maxima: grid (column blocks of 128, row chunks), a thread owns four columns
// and walks its rows eight apart, as the other row kernels of the step do.
constexpr int SPLIT_LANES_Y = 8;
__global__ void __launch_bounds__(32 * SPLIT_LANES_Y)
    split_rows_kernel(const float *__restrict__ x, int rows, int cols, int rows_per_chunk, PlaneSink k) {
  pdl_enter();
  __shared__ unsigned shared[SPLIT_LANES_Y * 128];
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  const int col = blockIdx.x * 128 + tx * 4;
  const bool live = col < cols;
  const float s = sink_scale(k);
  LineTracker track;
  if (live) {
    const int r0 = blockIdx.y * rows_per_chunk, r1 = min(rows, r0 + rows_per_chunk);
    for (int r = r0 + ty; r < r1; r += 2 * SPLIT_LANES_Y) {
      const int r2 = r + SPLIT_LANES_Y;
      const size_t o = (size_t)r * cols + col, o2 = (size_t)r2 * cols + col;
      const float4 v = __ldg(reinterpret_cast<const float4 *>(x + o));
      float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r2 < r1) w = __ldg(reinterpret_cast<const float4 *>(x + o2));
      const float a[4] = {v.x, v.y, v.z, v.w};
      sink_store4(k, o, a, s);
      track.row(k, r, a);
      if (r2 < r1) {
        const float b[4] = {w.x, w.y, w.z, w.w};
        sink_store4(k, o2, b, s);
        track.row(k, r2, b);
      }
    }
  }
  // Under a predicted scale the tensor's maximum is found here as well; where it
  // was known before (it gave s) the atomic maximum changes nothing.
  track.finish(k, shared, tx, ty, SPLIT_LANES_Y, blockIdx.x * 128, cols, live);
}

// Planes made for one product, of up to two operands in one launch, every line along
// the free dimension with the scale of its own maximum (so no line is small for its
// scale and the range guard has only infinities and NaN to flag).
//
// A line that is contiguous belongs to a warp: 1024 elements stay in its registers
// between the maximum and the split, the rest is read again.  Lines across the
// memory's rows (the mn-contiguous operands of the backward products) belong to a
// cluster: 64 columns, each CTA an eighth of the rows, the column maxima folded over
// the CTAs through their shared memory.  So every element comes from memory once
// and the second reading from L1.  Bound by memory latency at the sizes of the
// products that take it: 6 - 8 us for 3 M elements (24 MB, 3.5 TB/s) in L2, where a
// maximum, a split and a check per operand took 40.
constexpr int LS_THREADS = 256, LS_KEEP = 8, LS_COLS = 64, LS_CLUSTER = 8;
// Bits of 2^100.  Larger lines, infinities and NaN go to the fp32 path: the sums times
// such a line's 1 / scale would leave the range before the other factor brings them back.
constexpr unsigned LS_HUGE = (127u + 100u) << 23;

struct LineSplit {
  const float *x;
  long long pitch;      // of the rows in memory
  int rows, cols;       // in memory
  int by_columns;       // lines are columns
  int vec;              // rows allow 16-byte loads
  uint16_t *hi, *lo;
  long long out_pitch;  // of the planes' rows, a multiple of 8
  float *line_inv;      // 1 / scale of every line
  int blocks;
};

__device__ __forceinline__ float4 line_load4(const LineSplit &o, int row, int col) {
  const float *p = o.x + (long long)row * o.pitch + col;
  if (o.vec && col + 3 < o.cols) return __ldg(reinterpret_cast<const float4 *>(p));
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (col < o.cols) v.x = __ldg(p);
  if (col + 1 < o.cols) v.y = __ldg(p + 1);
  if (col + 2 < o.cols) v.z = __ldg(p + 2);
  if (col + 3 < o.cols) v.w = __ldg(p + 3);
  return v;
}
__device__ __forceinline__ unsigned abs_bits4(float4 v) {
  return max(max(abs_bits(v.x), abs_bits(v.y)), max(abs_bits(v.z), abs_bits(v.w)));
}
__device__ __forceinline__ void line_store4(const LineSplit &o, int row, int col, float4 v, float4 s) {
  PlaneSink k;
  k.hi = o.hi, k.lo = o.lo;
  const float t[4] = {v.x * s.x, v.y * s.y, v.z * s.z, v.w * s.w};  // exact
  sink_store4(k, (size_t)row * o.out_pitch + col, t, 1.f);
}

__device__ __forceinline__ void split_contiguous_lines(const LineSplit &o, int block, unsigned *flag) {
  const int row = block * (LS_THREADS / 32) + (int)threadIdx.x / 32, lane = threadIdx.x % 32;
  if (row >= o.rows) return;
  float4 v[LS_KEEP];
  unsigned m = 0u;
#pragma unroll
  for (int i = 0; i < LS_KEEP; ++i) {
    const int col = lane * 4 + i * 128;
    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (col < o.cols) v[i] = line_load4(o, row, col);
  }
#pragma unroll
  for (int i = 0; i < LS_KEEP; ++i) m = max(m, abs_bits4(v[i]));
#pragma unroll 4
  for (int col = lane * 4 + LS_KEEP * 128; col < o.cols; col += 128) m = max(m, abs_bits4(line_load4(o, row, col)));
  m = __reduce_max_sync(0xffffffffu, m);
  const float s = plane_scale_from_bits(m, PLANE_EXP_OWN);
  const float4 s4 = make_float4(s, s, s, s);
#pragma unroll
  for (int i = 0; i < LS_KEEP; ++i) {
    const int col = lane * 4 + i * 128;
    if (col < o.cols) line_store4(o, row, col, v[i], s4);
  }
#pragma unroll 4
  for (int col = lane * 4 + LS_KEEP * 128; col < o.cols; col += 128) line_store4(o, row, col, line_load4(o, row, col), s4);
  if (lane == 0) {
    o.line_inv[row] = 1.f / s;
    if (m >= LS_HUGE) atomicOr(flag, GUARD_WHOLE);
  }
}

__device__ __forceinline__ void split_column_lines(const LineSplit &o, int block, unsigned *flag) {
  __shared__ uint4 fold[LS_THREADS / 16][LS_COLS / 4];
  __shared__ unsigned cmax[LS_COLS];
  __shared__ float scale[LS_COLS];
  const int rank = block % LS_CLUSTER, col0 = block / LS_CLUSTER * LS_COLS;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16, col = col0 + tx * 4;
  const int r0 = (int)((long long)o.rows * rank / LS_CLUSTER) + ty, r1 = (int)((long long)o.rows * (rank + 1) / LS_CLUSTER);
  constexpr int STEP = LS_THREADS / 16;
  float4 v[LS_KEEP];
  uint4 m = make_uint4(0u, 0u, 0u, 0u);
  auto take = [&](float4 x) {
    m.x = max(m.x, abs_bits(x.x)), m.y = max(m.y, abs_bits(x.y));
    m.z = max(m.z, abs_bits(x.z)), m.w = max(m.w, abs_bits(x.w));
  };
#pragma unroll
  for (int i = 0; i < LS_KEEP; ++i) {
    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r0 + i * STEP < r1 && col < o.cols) v[i] = line_load4(o, r0 + i * STEP, col);
  }
#pragma unroll
  for (int i = 0; i < LS_KEEP; ++i) take(v[i]);
  if (col < o.cols) {
#pragma unroll 4
    for (int r = r0 + LS_KEEP * STEP; r < r1; r += STEP) take(line_load4(o, r, col));
  }
  fold[ty][tx] = m;
  __syncthreads();
  if (threadIdx.x < LS_COLS) {
    const unsigned *f = reinterpret_cast<const unsigned *>(fold);
    unsigned w = 0u;
#pragma unroll
    for (int y = 0; y < LS_THREADS / 16; ++y) w = max(w, f[y * LS_COLS + threadIdx.x]);
    cmax[threadIdx.x] = w;
  }
  tc::cluster_sync_all();
  if (threadIdx.x < LS_COLS) {
    unsigned w = 0u;
#pragma unroll
    for (int r = 0; r < LS_CLUSTER; ++r) {
      unsigned u;
      asm volatile("ld.shared::cluster.u32 %0, [%1];"
                   : "=r"(u)
                   : "r"(tc::map_to_cta(tc::smem_u32(cmax + threadIdx.x), (uint32_t)r)));
      w = max(w, u);
    }
    const float s = plane_scale_from_bits(w, PLANE_EXP_OWN);
    scale[threadIdx.x] = s;
    if (rank == 0 && col0 + (int)threadIdx.x < o.cols) {
      o.line_inv[col0 + threadIdx.x] = 1.f / s;
      if (w >= LS_HUGE) atomicOr(flag, GUARD_WHOLE);
    }
  }
  tc::cluster_sync_all();  // scales are set; no CTA leaves while another reads its maxima
  if (col >= o.out_pitch) return;
  const float4 s4 = *reinterpret_cast<const float4 *>(scale + tx * 4);
#pragma unroll
  for (int i = 0; i < LS_KEEP; ++i)
    if (r0 + i * STEP < r1) line_store4(o, r0 + i * STEP, col, v[i], s4);
#pragma unroll 4
  for (int r = r0 + LS_KEEP * STEP; r < r1; r += STEP) line_store4(o, r, col, line_load4(o, r, col), s4);
}

// Blocks [0, a.blocks) work on a, the rest on b.  flag: set where an operand holds a
// value the halves cannot stand for; next_flag: the word of the launch after this one.
__global__ void __launch_bounds__(LS_THREADS) split_lines_kernel(const __grid_constant__ LineSplit a,
                                                                 const __grid_constant__ LineSplit b, unsigned *flag,
                                                                 unsigned *next_flag) {
  pdl_enter();
  if (blockIdx.x == 0 && threadIdx.x == 0) *next_flag = 0u;
  const bool second = (int)blockIdx.x >= a.blocks;
  const LineSplit &o = second ? b : a;
  const int block = second ? (int)blockIdx.x - a.blocks : (int)blockIdx.x;
  if (o.by_columns) split_column_lines(o, block, flag);
  else split_contiguous_lines(o, block, flag);
}

// A block per tensor.
struct FinalizeBatch {
  PlaneSink sinks[UPDATE_BATCH];
};
__global__ void __launch_bounds__(1024) planes_finalize_kernel(const __grid_constant__ PlaneSink k) {
  pdl_enter(); sink_finalize(k); }
__global__ void __launch_bounds__(1024) planes_finalize_all_kernel(const __grid_constant__ FinalizeBatch b) {
  pdl_enter(); sink_finalize(b.sinks[blockIdx.x]); }

int stream_blocks(dlb_ctx *ctx, size_t items) {
  const size_t blocks = (items + 255) / 256;
  return (int)max((size_t)1, min(blocks, (size_t)ctx->sm_count * 16));
}

dlb_status scale_slot(dlb_ctx *ctx, float **out) {
  if (!ctx->scale_pool) {
    DLB_CUDA(cudaMalloc(&ctx->scale_pool, (size_t)SCALE_SLOTS * SLOT_WORDS * sizeof(float)));
    ctx->scale_free.reserve(SCALE_SLOTS);
    for (int i = SCALE_SLOTS - 1; i >= 0; --i) ctx->scale_free.push_back(i);
  }
  if (ctx->scale_free.empty()) {
    set_error("dlb_split_planes: more than %d plane buffers are registered", SCALE_SLOTS);
    return DLB_ERR_INVALID;
  }
  *out = ctx->scale_pool + (size_t)SLOT_WORDS * ctx->scale_free.back();
  ctx->scale_free.pop_back();
  return DLB_OK;
}

dlb_status guard_counters(dlb_ctx *ctx) {
  if (ctx->d_guard) return DLB_OK;
  DLB_CUDA(cudaMalloc(&ctx->d_guard, 4 * sizeof(unsigned long long)));
  DLB_CUDA(cudaMemsetAsync(ctx->d_guard, 0, 4 * sizeof(unsigned long long), ctx->stream));
  return DLB_OK;
}

void release_entry(dlb_ctx *ctx, dlb_ctx::PlaneEntry &e) {
  ctx->scale_free.push_back((int)((e.scale - ctx->scale_pool) / SLOT_WORDS));
  if (e.lines) {
    cudaStreamSynchronize(ctx->stream);  // a check kernel may still read the array
    cudaFree(e.lines);
    e.lines = nullptr;
  }
}

// The split pass of a tensor whose maximum is in its slot (or whose predicted
// scale is to be used): by rows with statistics where the shape allows.
dlb_status launch_split(dlb_ctx *ctx, const float *x, size_t n, int rows, int cols, const PlaneSink &k) {
  const bool by_rows = rows > 0 && cols > 0 && (cols & 3) == 0 && (size_t)rows * cols == n &&
                       ((reinterpret_cast<uintptr_t>(x) & 15) | (reinterpret_cast<uintptr_t>(k.hi) & 7) |
                        (reinterpret_cast<uintptr_t>(k.lo) & 7)) == 0;
  if (by_rows) {
    const int col_blocks = ceil_div(cols, 128);
    int chunks = max(1, min(ceil_div(ctx->sm_count * 8, col_blocks), ceil_div(rows, 2 * SPLIT_LANES_Y)));
    const int rpc = ceil_div(ceil_div(rows, chunks), 2 * SPLIT_LANES_Y) * 2 * SPLIT_LANES_Y;
    chunks = ceil_div(rows, rpc);
    DLB_LAUNCH_KERNEL(ctx, split_rows_kernel, dim3(col_blocks, chunks), 32 * SPLIT_LANES_Y, 0, x, rows, cols, rpc, k);
  } else {
    PlaneSink flat = k;
    flat.rowmax = flat.colmax = flat.lines = nullptr;
    flat.n_lines = flat.n_rows = 0;
    DLB_LAUNCH_KERNEL(ctx, split_flat_kernel, stream_blocks(ctx, n / 4 + 1), 256, 0, x, n, flat);
  }
  DLB_LAUNCHED(ctx);
  return DLB_OK;
}

}  // namespace

static size_t line_rows(const GemmOperand &o, int mn, int k) { return o.stride_k == 1 ? mn : k; }
static long long line_pitch(const GemmOperand &o, int mn, int k) {
  return (long long)align_up((size_t)(o.stride_k == 1 ? k : mn), 8);
}

dlb_status planes_split_lines(dlb_ctx *ctx, GemmOperand *A, int M, GemmOperand *B, int N, int K) {
  GemmOperand *const o[2] = {A, B};
  const int mn[2] = {M, N};
  size_t plane[2] = {0, 0}, halves = 0, lines = 0;
  for (int i = 0; i < 2; ++i)
    if (o[i]) {
      plane[i] = align_up(line_rows(*o[i], mn[i], K) * (size_t)line_pitch(*o[i], mn[i], K), 64);
      halves += 2 * plane[i];
      lines += align_up((size_t)mn[i], 4);
    }
  if (!ctx->line_flags) {
    DLB_CUDA(cudaMalloc(&ctx->line_flags, 2 * sizeof(unsigned)));
    DLB_CUDA(cudaMemsetAsync(ctx->line_flags, 0, 2 * sizeof(unsigned), ctx->stream));
  }
  void *scr = nullptr;
  DLB_TRY(scratch(ctx, halves * sizeof(uint16_t) + lines * sizeof(float), &scr));
  uint16_t *h = static_cast<uint16_t *>(scr);
  float *inv = reinterpret_cast<float *>(h + halves);
  unsigned *flag = ctx->line_flags + (ctx->line_splits & 1), *next = ctx->line_flags + (~ctx->line_splits & 1);
  ctx->line_splits++;
  LineSplit job[2] = {};
  bool columns = false;
  for (int i = 0; i < 2; ++i)
    if (o[i]) {
      LineSplit &j = job[i];
      GemmOperand &op = *o[i];
      const bool by_rows = op.stride_k == 1;
      j.x = op.ptr;
      j.pitch = by_rows ? op.stride_mn : op.stride_k;
      j.rows = by_rows ? mn[i] : K;
      j.cols = by_rows ? K : mn[i];
      j.by_columns = by_rows ? 0 : 1;
      j.vec = (reinterpret_cast<uintptr_t>(j.x) & 15) == 0 && (j.pitch & 3) == 0;
      j.hi = h;
      j.lo = h + plane[i];
      j.out_pitch = line_pitch(op, mn[i], K);
      j.line_inv = inv;
      j.blocks = by_rows ? (int)align_up((size_t)ceil_div(j.rows, LS_THREADS / 32), LS_CLUSTER)
                         : LS_CLUSTER * (int)((j.out_pitch + LS_COLS - 1) / LS_COLS);
      columns |= !by_rows;
      op.fp32_stride_mn = op.stride_mn;
      op.fp32_stride_k = op.stride_k;
      (by_rows ? op.stride_mn : op.stride_k) = j.out_pitch;
      op.h_hi = j.hi;
      op.h_lo = j.lo;
      op.scale = op.line_inv = inv;
      op.guard = flag;
      op.guard_mask = GUARD_WHOLE;
      h += 2 * plane[i];
      inv += align_up((size_t)mn[i], 4);
    }
  const unsigned grid = (unsigned)(job[0].blocks + job[1].blocks);
  if (columns) {
    DLB_CUDA(launch_kernel_cluster(ctx, split_lines_kernel, dim3(grid), dim3(LS_THREADS), 0, LS_CLUSTER, job[0], job[1],
                                   flag, next));
  } else {
    DLB_LAUNCH_KERNEL(ctx, split_lines_kernel, grid, LS_THREADS, 0, job[0], job[1], flag, next);
  }
  DLB_LAUNCHED(ctx);
  ctx->products[DLB_PRODUCT_FRESH_PLANES]++;
  return DLB_OK;
}

void planes_rows_exempt(dlb_ctx *ctx, const float *planes, size_t bytes, bool on) {
  if (!planes) return;
  const uintptr_t key = reinterpret_cast<uintptr_t>(planes);
  if (on && !ctx->guard_strict) ctx->rows_exempt[key] = bytes;
  else ctx->rows_exempt.erase(key);
}

// Whether a plane buffer starting at `key` lies inside a marked one.
static bool rows_exempt_at(const dlb_ctx *ctx, uintptr_t key) {
  auto it = ctx->rows_exempt.upper_bound(key);
  if (it == ctx->rows_exempt.begin()) return false;
  --it;
  return key < it->first + it->second;
}

void planes_unused(dlb_ctx *ctx, const float *planes, size_t bytes, bool on) {
  if (!planes) return;
  const uintptr_t key = reinterpret_cast<uintptr_t>(planes);
  if (on) ctx->planes_unused[key] = bytes;
  else ctx->planes_unused.erase(key);
}

bool planes_unused_at(const dlb_ctx *ctx, const float *planes) {
  if (ctx->planes_unused.empty()) return false;
  const uintptr_t key = reinterpret_cast<uintptr_t>(planes);
  auto it = ctx->planes_unused.upper_bound(key);
  if (it == ctx->planes_unused.begin()) return false;
  --it;
  return key < it->first + it->second;
}

bool planes_lookup(dlb_ctx *ctx, const float *aux, GemmOperand *o) {
  if (!aux || ctx->planes.empty() || planes_unused_at(ctx, aux)) return false;
  const uintptr_t p = reinterpret_cast<uintptr_t>(aux);
  auto it = ctx->planes.upper_bound(p);
  if (it == ctx->planes.begin()) return false;
  --it;
  const dlb_ctx::PlaneEntry &e = it->second;
  if (p >= it->first + e.n * sizeof(float)) return false;
  const size_t off = (p - it->first) / sizeof(float);
  if (e.x + off != o->ptr) return false;  // the buffer belongs to another tensor
  const uint16_t *hi = reinterpret_cast<const uint16_t *>(it->first) + off;
  const uint16_t *lo = hi + e.n;
  if ((reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 15) return false;
  o->h_hi = hi;
  o->h_lo = lo;
  o->scale = e.scale;
  o->guard = reinterpret_cast<const unsigned *>(e.scale) + SLOT_FLAGS;
  o->guard_mask = guard_mask_of(*o);
  return true;
}

// Points a sink at the line statistics of a [rows, cols] tensor; the rows of an
// exempt tensor are not recorded at all.
static void sink_lines(PlaneSink &k, unsigned *lines, int rows, int cols, bool exempt) {
  k.lines = lines;
  k.n_rows = lines ? rows : 0;
  k.n_lines = lines ? rows + cols : 0;
  k.rowmax = lines && !exempt ? lines : nullptr;
  k.colmax = lines ? lines + rows : nullptr;
  k.rows_exempt = exempt ? 1 : 0;
}

// Room for the line maxima of a [rows, cols] tensor; they are zero between splits.
static dlb_status entry_lines(dlb_ctx *ctx, dlb_ctx::PlaneEntry &e) {
  const size_t need = (size_t)e.rows + e.cols;
  if (e.rows == 0 || need <= e.line_words) return DLB_OK;
  if (e.lines) {
    DLB_CUDA(cudaStreamSynchronize(ctx->stream));  // a check kernel may still read the array
    DLB_CUDA(cudaFree(e.lines));
    e.lines = nullptr;
    e.line_words = 0;
  }
  DLB_CUDA(cudaMalloc(&e.lines, need * sizeof(unsigned)));
  e.line_words = need;
  DLB_CUDA(cudaMemsetAsync(e.lines, 0, need * sizeof(unsigned), ctx->stream));
  return DLB_OK;
}

// Registers `planes` as the plane buffer of x[0..n) with the given shape (0, 0:
// none) and fills the job.  A registration of the same tensor and width is kept, with
// its predicted scale, also where the number of rows differs (a longer last batch of an
// epoch: dropped, it cost a cudaFree, a cudaMalloc and the fused form of the producing
// kernel, twice an epoch for every tensor); anything else this buffer overlaps is stale
// and dropped.
dlb_status planes_open(dlb_ctx *ctx, const float *x, float *planes, size_t n, int rows, int cols,
                       bool kernel_can_fuse, PlaneJob *job) {
  DLB_REQUIRE(x && planes && n > 0 && n < ((size_t)1 << 40), "plane buffer: tensor, buffer and size");
  if (planes_unused_at(ctx, planes)) {
    *job = PlaneJob{};
    return DLB_OK;
  }
  if ((size_t)rows * (size_t)cols != n) rows = cols = 0;
  const uintptr_t key = reinterpret_cast<uintptr_t>(planes);
  planes_forget(ctx, key + 1, n * sizeof(float) - 1);
  auto before = ctx->planes.lower_bound(key);
  if (before != ctx->planes.begin()) {
    --before;
    if (before->first + before->second.n * sizeof(float) > key) planes_forget(ctx, before->first, 1);
  }
  auto it = ctx->planes.find(key);
  if (it != ctx->planes.end()) {
    dlb_ctx::PlaneEntry &e = it->second;
    const bool same = e.x == x && e.n == n && e.rows == rows && e.cols == cols;
    if (!same && e.x == x && e.cols == cols && e.rows > 0 && rows > 0) {
      e.n = n;
      e.rows = rows;
      DLB_TRY(entry_lines(ctx, e));
    } else if (!same) {
      planes_forget(ctx, key, 1);
      it = ctx->planes.end();
    }
  }
  if (it == ctx->planes.end()) {
    dlb_ctx::PlaneEntry e;
    e.x = x;
    e.n = n;
    e.rows = rows;
    e.cols = cols;
    DLB_TRY(scale_slot(ctx, &e.scale));
    DLB_CUDA(cudaMemsetAsync(e.scale, 0, SLOT_WORDS * sizeof(float), ctx->stream));
    DLB_TRY(entry_lines(ctx, e));
    it = ctx->planes.emplace(key, e).first;
  }
  dlb_ctx::PlaneEntry &e = it->second;
  static const bool fuse_enabled = [] {
    const char *v = getenv("DLB_PLANES_FUSED");
    return !(v && v[0] == '0');
  }();
  job->x = x;
  job->planes = planes;
  job->n = n;
  job->rows = rows;
  job->cols = cols;
  job->active = true;
  job->fused = kernel_can_fuse && e.seen && fuse_enabled && rows > 0 && (cols & 3) == 0 &&
               (reinterpret_cast<uintptr_t>(planes) & 7) == 0 && ((n * 2) & 7) == 0;
  DLB_TRY(guard_counters(ctx));
  job->sink = PlaneSink{};
  job->sink.slot = e.scale;
  job->sink.guard = ctx->d_guard;
  job->sink.rows_exempt = rows_exempt_at(ctx, key) ? 1 : 0;
  if (job->fused) {
    sink_lines(job->sink, e.lines, rows, cols, job->sink.rows_exempt != 0);
    job->sink.hi = reinterpret_cast<uint16_t *>(planes);
    job->sink.lo = job->sink.hi + n;
    job->sink.predicted = 1;
    job->sink.x = x;
    job->sink.n = n;
  }
  return DLB_OK;
}

dlb_status planes_close(dlb_ctx *ctx, const PlaneJob &job) {
  if (!job.active) return DLB_OK;
  auto it = ctx->planes.find(reinterpret_cast<uintptr_t>(job.planes));
  DLB_REQUIRE(it != ctx->planes.end(), "plane buffer: closed without a registration");
  dlb_ctx::PlaneEntry &e = it->second;
  if (!job.fused) {
    // The producing kernel left the tensor's maximum in the slot: the split pass.
    PlaneSink k;
    k.hi = reinterpret_cast<uint16_t *>(job.planes);
    k.lo = k.hi + job.n;
    k.slot = e.scale;
    sink_lines(k, e.lines, e.rows, e.cols, job.sink.rows_exempt != 0);
    k.predicted = 0;
    k.guard = ctx->d_guard;
    DLB_TRY(launch_split(ctx, job.x, job.n, e.rows, e.cols, k));
  }
  PlaneSink k = job.sink;
  sink_lines(k, e.lines, e.rows, e.cols, job.sink.rows_exempt != 0);
  k.predicted = job.fused ? 1 : 0;
  DLB_LAUNCH_KERNEL(ctx, planes_finalize_kernel, 1, 1024, 0, k);
  DLB_LAUNCHED(ctx);
  e.seen = true;
  return DLB_OK;
}

dlb_status planes_close_all(dlb_ctx *ctx, const PlaneJob *jobs, int count) {
  for (int first = 0; first < count; first += UPDATE_BATCH) {
    FinalizeBatch b;
    const int n = min(UPDATE_BATCH, count - first);
    for (int i = 0; i < n; ++i) {
      const PlaneJob &job = jobs[first + i];
      auto it = ctx->planes.find(reinterpret_cast<uintptr_t>(job.planes));
      DLB_REQUIRE(job.active && job.fused && it != ctx->planes.end(), "plane buffers: closed together");
      b.sinks[i] = job.sink;
      sink_lines(b.sinks[i], it->second.lines, it->second.rows, it->second.cols, job.sink.rows_exempt != 0);
      b.sinks[i].predicted = 1;
      it->second.seen = true;
    }
    DLB_LAUNCH_KERNEL(ctx, planes_finalize_all_kernel, n, 1024, 0, b);
    DLB_LAUNCHED(ctx);
  }
  return DLB_OK;
}

dlb_status planes_absmax(dlb_ctx *ctx, const float *x, size_t n, float *slot) {
  DLB_LAUNCH_KERNEL(ctx, absmax_kernel, stream_blocks(ctx, n / 4 + 1), 256, 0, x, n, reinterpret_cast<unsigned *>(slot) + SLOT_AMAX);
  DLB_LAUNCHED(ctx);
  return DLB_OK;
}

// Drops the entries whose buffer starts inside [base, base + bytes).
void planes_forget(dlb_ctx *ctx, uintptr_t base, size_t bytes) {
  auto it = ctx->planes.lower_bound(base);
  while (it != ctx->planes.end() && it->first < base + bytes) {
    release_entry(ctx, it->second);
    it = ctx->planes.erase(it);
  }
}

}  // namespace dlb

using namespace dlb;

extern "C" {

dlb_status dlb_ctx_set_gemm_kind(dlb_ctx *ctx, int kind) {
  DLB_REQUIRE(ctx && (kind == DLB_GEMM_TF32X3 || kind == DLB_GEMM_F16X3), "dlb_ctx_set_gemm_kind");
  if (kind == ctx->gemm_kind) return DLB_OK;
  // Plane buffers written under the other form do not hold what this form
  // reads: drop every registration and let the models split their weights
  // again (they compare plane_generation before each forward pass).
  DLB_CUDA(cudaStreamSynchronize(ctx->stream));
  planes_forget(ctx, 0, ~(size_t)0);
  ctx->plane_generation++;
  ctx->gemm_kind = kind;
  return DLB_OK;
}

int dlb_ctx_gemm_kind(dlb_ctx *ctx) { return ctx ? ctx->gemm_kind : -1; }

dlb_status dlb_split_planes_2d(dlb_ctx *ctx, const float *x, float *planes, int rows, int cols) {
  DLB_REQUIRE(ctx && x && planes && rows >= 0 && cols >= 0, "dlb_split_planes_2d");
  const size_t n = (size_t)rows * (size_t)cols;
  if (n == 0) return DLB_OK;
  if (ctx->gemm_kind == DLB_GEMM_TF32X3) return dlb_split_tf32(ctx, x, planes, n);
  PlaneJob job;
  DLB_TRY(planes_open(ctx, x, planes, n, rows, cols, true, &job));
  if (!job.active) return DLB_OK;
  // With a scale predicted from this buffer's previous split one pass does; the
  // first split takes the tensor's maximum first.
  if (job.fused) DLB_TRY(launch_split(ctx, x, n, rows, cols, job.sink));
  else DLB_TRY(planes_absmax(ctx, x, n, job.sink.slot));
  return planes_close(ctx, job);
}

dlb_status dlb_split_planes(dlb_ctx *ctx, const float *x, float *planes, size_t n) {
  DLB_REQUIRE(ctx && x && planes, "dlb_split_planes: null");
  if (n == 0) return DLB_OK;
  if (ctx->gemm_kind == DLB_GEMM_TF32X3) return dlb_split_tf32(ctx, x, planes, n);
  PlaneJob job;
  DLB_TRY(planes_open(ctx, x, planes, n, 0, 0, false, &job));
  if (!job.active) return DLB_OK;
  DLB_TRY(planes_absmax(ctx, x, n, job.sink.slot));
  return planes_close(ctx, job);
}

dlb_status dlb_ctx_set_guard_strict(dlb_ctx *ctx, int strict) {
  DLB_REQUIRE(ctx, "dlb_ctx_set_guard_strict: null");
  ctx->guard_strict = strict != 0;
  if (ctx->guard_strict) ctx->rows_exempt.clear();
  return DLB_OK;
}

dlb_status dlb_ctx_guard_resplits(dlb_ctx *ctx, uint64_t *tensors_resplit) {
  DLB_REQUIRE(ctx && tensors_resplit, "dlb_ctx_guard_resplits: null");
  unsigned long long host = 0;
  if (ctx->d_guard) {
    DLB_CUDA(cudaMemcpyAsync(&host, ctx->d_guard + 2, sizeof(host), cudaMemcpyDeviceToHost, ctx->stream));
    DLB_CUDA(cudaStreamSynchronize(ctx->stream));
  }
  *tensors_resplit = host;
  return DLB_OK;
}

dlb_status dlb_ctx_guard_counters(dlb_ctx *ctx, uint64_t *tensors_flagged, uint64_t *products_on_fallback) {
  DLB_REQUIRE(ctx && tensors_flagged && products_on_fallback, "dlb_ctx_guard_counters: null");
  unsigned long long host[2] = {0, 0};
  if (ctx->d_guard) {
    DLB_CUDA(cudaMemcpyAsync(host, ctx->d_guard, sizeof(host), cudaMemcpyDeviceToHost, ctx->stream));
    DLB_CUDA(cudaStreamSynchronize(ctx->stream));
  }
  *tensors_flagged = host[0];
  *products_on_fallback = host[1];
  return DLB_OK;
}

}  // extern "C"
