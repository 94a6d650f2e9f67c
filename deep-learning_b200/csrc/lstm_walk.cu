// The walk of an LSTM layer over time in one launch per direction.
//
// Step by step (lstm.cu) a time step is a product of B rows with the recurrent
// weights and a kernel for the cells: two launches and two round trips through
// L2 of 15 - 20 us together, 32 steps x 2 layers x 2 directions in a pass of 2.2 ms.
// The examples of a batch are independent, though.  Here a cluster of CTAs takes
// up to EX examples through all T steps with the recurrent weights on the chip:
// CTA r of the CS holds the rows of its blocks (forward: the K + 3 rows of each
// block, [rows, C]; backward: the columns of its cells, [cells, G]), forms
// the sums of those rows for the EX examples in fp32, runs its cells, and sends
// their outputs (backward: their gates' errors) into every CTA's copy of the vector
// that the next step contracts with.  State (c, and backward the error of the state
// and of the gates) stays in registers of the thread that owns the (example, block).
//
// The exchange is by st.async onto an mbarrier that counts the bytes of a step, not
// by stores and a cluster barrier: the barrier's release waits until this step's
// stores to global memory are visible too, 6 us a step in all where this form takes
// 2.5 forward and 2.9 backward (64 examples, 128 blocks of 2 cells).  What bounds a step
// is one chain: inputs, the sums (about 115 cycles per example and 128 k), five squashing
// functions in a row, the exchange; all but the sums take 2800 cycles of the 4700 (the
// fit in plan_walk).  The copies and their barriers alternate: a
// CTA sends its part of step t + 2 only after it has all of step t + 1, so every
// other CTA has read step t by then.
//
// A warp forms the sums of ROWS rows: its lanes share 128 consecutive k, 512
// contiguous bytes of each row and of the vectors (128-bit loads of a quarter of a
// warp take a shared-memory cycle each even where quarters read the same address:
// with eight lanes to a row a step's sums took 3700 cycles, not 1600), and the
// sums over the lanes are formed by exchanging halves of the ROWS x EX values.  Where
// ROWS x k fits in the registers (CHUNKS) the weights stay there; otherwise they are
// read from shared memory, once per step for all EX examples.  One lane per cell does
// the rest; the lanes of a block exchange the peephole sums by shuffles.
#include <algorithm>

#include "common.cuh"
#include "lstm_cell.cuh"
#include "tc_pair.cuh"

namespace dlb {

namespace {

constexpr int W_THREADS = 512;  // 128 registers each
constexpr int W_MAX_CLUSTER = 8;

__host__ __device__ __forceinline__ int pad128(int n) { return (n + 127) & ~127; }

struct WalkShape {
  int rows, T, B, K;  // examples, time steps, blocks, cells per block
  int kp;             // K rounded up to a power of two: lanes of a block
  int cs;             // CTAs of a cluster
  int *status;
};

// Two products and sums at once (each rounded as by fmaf).
__device__ __forceinline__ void fma2(uint64_t &d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum2(uint64_t v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  return (uint64_t)__float_as_uint(a) | (uint64_t)__float_as_uint(b) << 32;
}
// A load that stays where it is written: the step's inputs are fetched before the
// wait for the other CTAs, not after it.
__device__ __forceinline__ float load_now(const float *p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}

// Sums N values over the lanes of a warp, each value ending up in one lane: at
// every level a lane keeps one half of the values and gives the other away.
template <int N, int MASK>
__device__ __forceinline__ void lane_sums(float *v, int lane) {
  if constexpr (MASK > 0) {
    constexpr int H = (N + 1) / 2;
    const bool up = lane & MASK;
#pragma unroll
    for (int i = 0; i < H; ++i) {
      if constexpr (N == 1) {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], MASK);
      } else {
        const float hi = i + H < N ? v[i + H] : 0.f;
        const float got = __shfl_xor_sync(0xffffffffu, up ? v[i] : hi, MASK);
        v[i] = (up ? hi : v[i]) + got;
      }
    }
    lane_sums<H, MASK / 2>(v, lane);
  }
}
// Which of the N values this lane holds afterwards, -1: none.
__device__ __forceinline__ int lane_sums_index(int n, int lane) {
  int index = 0, count = n;
  for (int m = 16; m > 0; m /= 2) {
    const bool up = lane & m;
    if (n == 1) {
      if (up) count = 0;
      continue;
    }
    const int h = (n + 1) / 2;
    index += up ? h : 0;
    count = up ? count - h : min(count, h);
    n = h;
  }
  return count > 0 ? index : -1;
}

// The sums of this CTA's rows: sums[row][e] = sum_k w[row][k] v[e][k]; k is padded to
// a multiple of 128 with zeros.  CHUNKS > 0: warp i holds rows [i ROWS, i ROWS + ROWS)
// in registers, at most CHUNKS x 128 k.
template <int EX, int ROWS, int CHUNKS>
struct RowSums {
  ulonglong2 reg[CHUNKS ? ROWS * CHUNKS : 1];
  const float *w;
  int pitch, rows, index;

  // load(row, k): the weights as they lie in global memory, zero beyond them.
  template <class Load>
  __device__ __forceinline__ void init(float *smem_w, int pitch_, int rows_, bool rows_inner, Load load) {
    w = smem_w, pitch = pitch_, rows = rows_, index = lane_sums_index(ROWS * EX, threadIdx.x & 31);
    if constexpr (CHUNKS > 0) {
      const int r0 = (int)threadIdx.x / 32 * ROWS, k0 = (threadIdx.x & 31) * 4;
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int j = 0; j < CHUNKS; ++j) {
          float v[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) v[q] = r0 + r < rows && j * 128 < pitch ? load(r0 + r, j * 128 + k0 + q) : 0.f;
          reg[r * CHUNKS + j].x = pack2(v[0], v[1]);
          reg[r * CHUNKS + j].y = pack2(v[2], v[3]);
        }
    } else {
      for (int i = threadIdx.x; i < rows * pitch; i += blockDim.x) {
        const int r = rows_inner ? i % rows : i / pitch, k = rows_inner ? i / rows : i % pitch;
        smem_w[(size_t)r * pitch + k] = load(r, k);
      }
    }
  }

  __device__ __forceinline__ void run(const float *v, float *sums) const {
    const int lane = threadIdx.x & 31;
    const ulonglong2 *vr = reinterpret_cast<const ulonglong2 *>(v) + lane;
    const int step = pitch / 4;
    for (int r0 = (int)threadIdx.x / 32 * ROWS; r0 < rows; r0 += (int)blockDim.x / 32 * ROWS) {
      float s[ROWS * EX];
      if constexpr (CHUNKS > 0) {
#pragma unroll
        for (int e = 0; e < EX; ++e) {
          uint64_t acc[ROWS];
#pragma unroll
          for (int r = 0; r < ROWS; ++r) acc[r] = 0;
#pragma unroll
          for (int j = 0; j < CHUNKS; ++j)
            if (j * 128 < pitch) {
              const ulonglong2 b = vr[e * step + j * 32];
#pragma unroll
              for (int r = 0; r < ROWS; ++r) {
                fma2(acc[r], reg[r * CHUNKS + j].x, b.x);
                fma2(acc[r], reg[r * CHUNKS + j].y, b.y);
              }
            }
#pragma unroll
          for (int r = 0; r < ROWS; ++r) s[r * EX + e] = sum2(acc[r]);
        }
      } else {
        uint64_t acc[ROWS * EX];
#pragma unroll
        for (int i = 0; i < ROWS * EX; ++i) acc[i] = 0;
        const ulonglong2 *wr[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
          wr[r] = reinterpret_cast<const ulonglong2 *>(w + (size_t)min(r0 + r, rows - 1) * pitch) + lane;
        for (int k = 0; k < step; k += 32) {
          ulonglong2 a[ROWS];
#pragma unroll
          for (int r = 0; r < ROWS; ++r) a[r] = wr[r][k];
#pragma unroll
          for (int e = 0; e < EX; ++e) {
            const ulonglong2 b = vr[e * step + k];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
              fma2(acc[r * EX + e], a[r].x, b.x);
              fma2(acc[r * EX + e], a[r].y, b.y);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < ROWS * EX; ++i) s[i] = sum2(acc[i]);
      }
      lane_sums<ROWS * EX, 16>(s, lane);
      if (index >= 0) sums[r0 * EX + index] = s[0];
      if constexpr (CHUNKS > 0) break;
    }
  }
};

// tc::map_to_cta that the compiler may take out of a loop.
__device__ __forceinline__ uint32_t map_here(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// The vectors that the steps hand on: two copies [EX, pitch] in every CTA, each with
// a barrier that counts the bytes that arrive for it.
struct Exchange {
  float *copies;
  uint32_t bar;  // two mbarriers, 8 bytes apart
  int cs, size, bytes, *abort_flag, *status;

  __device__ __forceinline__ void init(float *at, uint64_t *bars, int *flag, int size_, int bytes_, int cs_, int *status_) {
    copies = at, bar = tc::smem_u32(bars), cs = cs_, size = size_, bytes = bytes_, abort_flag = flag, status = status_;
    for (int i = threadIdx.x; i < 2 * size; i += blockDim.x) copies[i] = 0.f;
    if (threadIdx.x == 0) {
      *abort_flag = 0;
      if (cs > 1) {
        tc::mbar_init(bar, 1);
        tc::mbar_init(bar + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tc::mbar_expect_tx(bar, (uint32_t)bytes);
        tc::mbar_expect_tx(bar + 8, (uint32_t)bytes);
      }
    }
    if (cs > 1) tc::cluster_sync_all();
    else __syncthreads();
  }
  __device__ __forceinline__ float *copy(int step) const { return copies + (step & 1) * size; }
  // One or two floats at `at` of copy `step`, in CTAs first, first + by, ...
  __device__ __forceinline__ void send(int step, int at, float v, int first, int by) const {
    if (cs == 1) {
      if (first == 0) copy(step)[at] = v;
      return;
    }
    const uint32_t to = (uint32_t)((copy(step) + at - copies) * 4), on = (step & 1) * 8;
    for (int r = first; r < cs; r += by)
      asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(
                       map_here(tc::smem_u32(copies), (uint32_t)r) + to), "r"(__float_as_uint(v)), "r"(map_here(bar, (uint32_t)r) + on)
                   : "memory");
  }
  __device__ __forceinline__ void send2(int step, int at, float a, float b, int first, int by) const {
    if (cs == 1) {
      if (first == 0) {
        copy(step)[at] = a;
        copy(step)[at + 1] = b;
      }
      return;
    }
    const uint32_t to = (uint32_t)((copy(step) + at - copies) * 4), on = (step & 1) * 8;
    for (int r = first; r < cs; r += by)
      asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(
                       map_here(tc::smem_u32(copies), (uint32_t)r) + to), "r"(__float_as_uint(a)), "r"(__float_as_uint(b)),
                   "r"(map_here(bar, (uint32_t)r) + on)
                   : "memory");
  }
  // All of copy `step` is here.  A wait that runs out sets the status; the walk goes
  // on without waiting.
  __device__ __forceinline__ void wait(int step) const {
    if (cs == 1) {
      __syncthreads();
      return;
    }
    if (!tc::mbar_wait_cluster(bar + (step & 1) * 8, (uint32_t)(step >> 1) & 1u, abort_flag, status)) return;
    if (threadIdx.x == 0) tc::mbar_expect_tx(bar + (step & 1) * 8, (uint32_t)bytes);
  }
  // No CTA leaves while another may still send to it; after a wait that ran out the
  // barrier says nothing about the values in flight.
  __device__ __forceinline__ void finish() const {
    if (cs > 1) {
      tc::cluster_sync_all();
      if (*static_cast<volatile int *>(abort_flag)) tc::drain_pause();
    }
  }
};

// The walk's shared memory, in floats.  rows: of the CTA with the most blocks, so that
// the parts lie at the same place in every CTA.
__host__ __device__ __forceinline__ size_t walk_weights(bool reg, int rows, int pitch) {
  return reg ? 0 : (size_t)rows * pitch;
}
__host__ __device__ __forceinline__ size_t walk_floats(int ex, bool reg, int rows, int pitch) {
  return walk_weights(reg, rows, pitch) + 2 * (size_t)ex * pitch + (size_t)(rows + 12) * ex;
}

// What the threads of a CTA own: thread (e, b, k) is cell k of block b0 + b of example
// e0 + e through all time steps; k < kp, a power of two.  Four lanes per cell, one for
// each squashing function of a round, were no faster: 95 us against 92.
template <int EX>
struct Owner {
  int b0, nb, nb_max, e, b, k, n, block, examples, kp;
  bool cell, warp;  // the thread owns a cell; some thread of its warp may
  __device__ __forceinline__ Owner(const WalkShape &s) {
    const int rank = s.cs == 1 ? 0 : (int)tc::cluster_rank(), e0 = (int)blockIdx.x / s.cs * EX;
    kp = s.kp;
    b0 = (int)((long long)s.B * rank / s.cs);
    nb = (int)((long long)s.B * (rank + 1) / s.cs) - b0;
    nb_max = (s.B + s.cs - 1) / s.cs;
    k = (int)threadIdx.x & (kp - 1);
    const int q = (int)threadIdx.x / kp;
    e = q / nb, b = q - e * nb;
    n = e0 + e, block = b0 + b;
    examples = min(EX, s.rows - e0);
    cell = e < examples && k < s.K;
    warp = (int)(threadIdx.x & ~31u) / kp < EX * nb;
  }
  // Over the cells of the block, in all its lanes.
  __device__ __forceinline__ float sum(float x) const {
    x = cell ? x : 0.f;
    for (int m = kp / 2; m > 0; m /= 2) x += __shfl_xor_sync(0xffffffffu, x, m);
    return x;
  }
  // The value of a cell into every CTA's copy: the lanes of a pair of cells
  // send both values, each to half of the CTAs.
  __device__ __forceinline__ void send_cell(const Exchange &x, int step, int at, float v, int K) const {
    if (K % 2 == 0) {
      const float other = __shfl_xor_sync(0xffffffffu, v, 1);
      const int odd = k & 1;
      if (cell) x.send2(step, at + k - odd, odd ? other : v, odd ? v : other, odd, 2);
    } else if (cell) {
      x.send(step, at + k, v, 0, 1);
    }
  }
};

struct ForwardWalk {
  WalkShape s;
  const float *g_in;   // [T, rows, G]
  const float *w_rec;  // [G, C]
  const float *bias, *peep;
  float *z, *c, *ca, *h, *gi, *gf, *go;
};

template <int EX, int ROWS, int CHUNKS>
__global__ void __launch_bounds__(W_THREADS, 1) lstm_forward_walk_kernel(const __grid_constant__ ForwardWalk a) {
  extern __shared__ __align__(16) float walk_smem[];
  __shared__ uint64_t bars[2];
  __shared__ int abort_flag;
  pdl_enter();
  const Owner<EX> me(a.s);
  const int B = a.s.B, K = a.s.K, C = B * K, G = C + 3 * B, pitch = pad128(C), nb = me.nb;
  // Row order: the cells of all my blocks, then i, f, o of every block.
  RowSums<EX, ROWS, CHUNKS> rows;
  rows.init(walk_smem, pitch, nb * (K + 3), false, [&](int r, int k) {
    const int g = r < nb * K ? me.b0 * K + r : C + ((r - nb * K) / nb) * B + me.b0 + (r - nb * K) % nb;
    return k < C ? __ldg(a.w_rec + (size_t)g * C + k) : 0.f;
  });
  Exchange hv;
  hv.init(walk_smem + walk_weights(CHUNKS > 0, me.nb_max * (K + 3), pitch), bars, &abort_flag, EX * pitch,
          me.examples * C * 4, a.s.cs, a.s.status);
  float *sums = hv.copies + 2 * EX * pitch;

  const int cc = me.block * K + me.k;
  float bz = 0.f, bi = 0.f, bf = 0.f, bo = 0.f, pi = 0.f, pf = 0.f, po = 0.f;
  if (me.cell) {
    bz = __ldg(a.bias + cc), bi = __ldg(a.bias + C + me.block), bf = __ldg(a.bias + C + B + me.block);
    bo = __ldg(a.bias + C + 2 * B + me.block);
    pi = __ldg(a.peep + cc), pf = __ldg(a.peep + C + cc), po = __ldg(a.peep + 2 * C + cc);
  }
  float c = 0.f;
  for (int t = 0; t < a.s.T; ++t) {
    const size_t row = (size_t)t * a.s.rows + me.n;
    float sz = 0.f, si = 0.f, sf = 0.f, so = 0.f;
    if (me.cell) {
      const float *g = a.g_in + row * G;
      sz = load_now(g + cc), si = load_now(g + C + me.block), sf = load_now(g + C + B + me.block);
      so = load_now(g + C + 2 * B + me.block);
    }
    if (t > 0) {
      hv.wait(t - 1);
      rows.run(hv.copy(t - 1), sums);
      __syncthreads();
      if (me.cell) {
        const float *s = sums + me.e;
        sz += s[(me.b * K + me.k) * EX];
        si += s[(nb * K + me.b) * EX];
        sf += s[(nb * K + nb + me.b) * EX];
        so += s[(nb * K + 2 * nb + me.b) * EX];
      }
    }
    if (me.warp) {
      // Gates: input + recurrent + bias + peepholes (fwp_rec_mp.cpp L:1041-1062); no
      // forget gate at the first step.
      si += bi;
      sf += bf;
      if (t > 0) {
        si += me.sum(c * pi);
        sf += me.sum(c * pf);
      }
      const float gate_i = sigmoid_ref(si), gate_f = t > 0 ? sigmoid_ref(sf) : 0.f, z = tanh_ref(sz + bz);
      c = z * gate_i + c * gate_f;
      const float ca = tanh_ref(c);
      // Peephole from the new state (L:1330-1336).
      const float gate_o = sigmoid_ref(so + bo + me.sum(c * po)), h = ca * gate_o;
      if (t + 1 < a.s.T) me.send_cell(hv, t, me.e * pitch + me.block * K, h, K);
      if (me.cell) {
        const size_t at = row * C + cc;
        a.z[at] = z;
        a.c[at] = c;
        a.ca[at] = ca;
        a.h[at] = h;
        if (me.k == 0) {
          a.gi[row * B + me.block] = gate_i;
          a.gf[row * B + me.block] = gate_f;
          a.go[row * B + me.block] = gate_o;
        }
      }
    }
  }
  hv.finish();
}

struct BackwardWalk {
  WalkShape s;
  float *dH;           // [T, rows, C] error of the outputs from above; the recurrent part is added
  const float *w_rec;  // [G, C]
  const float *z, *ca, *c, *gi, *gf, *go, *peep;
  float *d;            // [T, rows, G]
};

// The gates' errors in the vector that the steps hand on: dz of every cell, then di
// and df of every block side by side, then do.
__host__ __device__ __forceinline__ int error_pitch(int B, int K) { return pad128(((B * K + 1) & ~1) + 3 * B); }

template <int EX, int ROWS, int CHUNKS>
__global__ void __launch_bounds__(W_THREADS, 1) lstm_backward_walk_kernel(const __grid_constant__ BackwardWalk a) {
  extern __shared__ __align__(16) float walk_smem[];
  __shared__ uint64_t bars[2];
  __shared__ int abort_flag;
  pdl_enter();
  const Owner<EX> me(a.s);
  const int B = a.s.B, K = a.s.K, C = B * K, G = C + 3 * B, C2 = (C + 1) & ~1, pitch = error_pitch(B, K);
  RowSums<EX, ROWS, CHUNKS> rows;
  rows.init(walk_smem, pitch, me.nb * K, true, [&](int r, int k) {
    int g = k;
    if (k >= C2 + 2 * B) g = k - C2 + C;
    else if (k >= C2) g = C + ((k - C2) & 1) * B + (k - C2) / 2;
    else if (k >= C) return 0.f;
    return g < G ? __ldg(a.w_rec + (size_t)g * C + me.b0 * K + r) : 0.f;
  });
  Exchange dv;
  dv.init(walk_smem + walk_weights(CHUNKS > 0, me.nb_max * K, pitch), bars, &abort_flag, EX * pitch,
          me.examples * G * 4, a.s.cs, a.s.status);
  float *sums = dv.copies + 2 * EX * pitch;

  const int cc = me.block * K + me.k;
  float pi = 0.f, pf = 0.f, po = 0.f;
  if (me.cell) pi = __ldg(a.peep + cc), pf = __ldg(a.peep + C + cc), po = __ldg(a.peep + 2 * C + cc);
  // Of the step after: state error, gates' errors, forget gate.
  float dC = 0.f, d_i = 0.f, d_f = 0.f, f_next = 0.f;
  for (int step = 0; step < a.s.T; ++step) {
    const int t = a.s.T - 1 - step;
    const size_t row = (size_t)t * a.s.rows + me.n, at = row * C + cc;
    float dH = 0.f, z = 0.f, ca = 0.f, c_prev = 0.f, gate_i = 0.f, gate_f = 0.f, gate_o = 0.f;
    if (me.cell) {
      dH = load_now(a.dH + at), z = load_now(a.z + at), ca = load_now(a.ca + at);
      if (t > 0) c_prev = load_now(a.c + at - (size_t)a.s.rows * C);
      gate_i = load_now(a.gi + row * B + me.block), gate_f = load_now(a.gf + row * B + me.block);
      gate_o = load_now(a.go + row * B + me.block);
    }
    if (step > 0) {
      dv.wait(step - 1);
      rows.run(dv.copy(step - 1), sums);
      __syncthreads();
      if (me.cell) dH += sums[(me.b * K + me.k) * EX + me.e];
    }
    if (me.warp) {
      // Output gate (bwp_rec_mp.cpp L:1199-1212); then the cell state: through the
      // output, the three peepholes and the next state (L:1257-1309, L:1372-1384).
      const float d_o = gate_o * (1.f - gate_o) * me.sum(dH * ca);
      float e = dH * gate_o * (1.f - ca * ca);
      e += po * d_o;
      e += pi * d_i;
      e += pf * d_f;
      e += dC * f_next;
      dC = e;
      f_next = gate_f;
      const float dz = e * gate_i * (1.f - z * z);
      d_i = me.sum(e * z) * gate_i * (1.f - gate_i);
      d_f = me.sum(e * c_prev) * gate_f * (1.f - gate_f);  // zero at t = 0: no forget gate (L:1440-1500)
      if (t > 0) {
        const int v = me.e * pitch;
        me.send_cell(dv, step, v + me.block * K, dz, K);
        if (me.cell) {
          dv.send2(step, v + C2 + 2 * me.block, d_i, d_f, me.k, K);
          dv.send(step, v + C2 + 2 * B + me.block, d_o, me.k, K);
        }
      }
      if (me.cell) {
        float *d = a.d + row * G;
        d[cc] = dz;
        if (step > 0) a.dH[at] = dH;
        if (me.k == 0) {
          d[C + me.block] = d_i;
          d[C + B + me.block] = d_f;
          d[C + 2 * B + me.block] = d_o;
        }
      }
    }
  }
  dv.finish();
}

// How a walk is laid out, and about how long it takes.
struct WalkPlan {
  int ex = 0, cs = 1, threads = 0;
  int form = 0;  // of W_FORMS
  size_t smem = 0;
  double us = 1e30;
};

constexpr size_t W_SMEM_MAX = 226 * 1024;  // beside the barriers

// Rows of a warp, and up to how many chunks of k its registers hold of them (0: the
// weights lie in shared memory).  A lane keeps ROWS x CHUNKS quads of weights beside the
// sums of ROWS x EX examples: about 10 quads, 40 of its 128 registers, leave room for 32
// sums, about 20 for 10, so those take more rows or a longer k but fewer examples.  Either
// number is divided between rows and chunks in the ways that some layer measured fastest
// with: 79 layers of 8 - 300 blocks of 1 - 3 cells at 8, 64 and 200 examples, every plan
// of both directions.  (4 x 5, 5 x 4, 1 x 10, 10 x 1 and 20 x 1 never won by more than 4 %.)
struct WarpRows {
  int rows, chunks;
};
constexpr WarpRows W_FORMS[] = {{5, 2}, {3, 3}, {2, 5}, {10, 2}, {6, 3}, {3, 6}, {2, 10}, {4, 0}};
constexpr int W_NUM_FORMS = sizeof(W_FORMS) / sizeof(W_FORMS[0]);
constexpr bool form_dense(int form) { return W_FORMS[form].rows * W_FORMS[form].chunks > 10; }
constexpr bool form_exists(int form, int ex) {
  return W_FORMS[form].rows * ex <= (form_dense(form) ? 10 : 32);
}

template <int EX, int FORM>
constexpr auto walk_kernel(const ForwardWalk &) {
  return lstm_forward_walk_kernel<EX, W_FORMS[FORM].rows, W_FORMS[FORM].chunks>;
}
template <int EX, int FORM>
constexpr auto walk_kernel(const BackwardWalk &) {
  return lstm_backward_walk_kernel<EX, W_FORMS[FORM].rows, W_FORMS[FORM].chunks>;
}

// Clusters of cs CTAs, one CTA to an SM, that run at once.
int walk_clusters(const dlb_ctx *ctx, int cs) {
  if (cs == 1) return ctx->sm_count;
  static int known[MAX_DEVICES][W_MAX_CLUSTER + 1] = {};
  int &n = known[ctx->device][cs];
  if (n == 0) n = resident_clusters(ctx, lstm_forward_walk_kernel<4, 4, 0>, W_THREADS, W_SMEM_MAX, cs);
  return n;
}

// The fastest layout by the cost of a step in cycles, fitted to the plans of the layers
// above near their fastest (the plan it picks takes 1.5 % longer than the fastest on
// average, 43 % at worst, 14 % next to it): cells and exchange; a chain of loads and multiply-adds per
// example and 128 k, times the rounds of rows per warp; the sums over lanes; the
// weights read from shared memory; and what the dense forms lose to spills.  Times the
// rounds that the examples need of the CTAs that run at once.  None if the weights do
// not fit.
WalkPlan plan_walk(const dlb_ctx *ctx, const WalkShape &s, int rows_per_block, int pitch) {
  WalkPlan best;
  if (s.kp > 32) return best;
  for (int cs = 1; cs <= W_MAX_CLUSTER && cs <= s.B; cs *= 2)
    for (int form = 0; form < W_NUM_FORMS; ++form)
      for (int ex : {1, 2, 4, 5, 8}) {
        if (!form_exists(form, ex)) continue;
        WalkPlan p;
        p.ex = ex, p.cs = cs, p.form = form;
        const int per_warp = W_FORMS[form].rows, chunks = W_FORMS[form].chunks;
        const int nb = ceil_div(s.B, cs), rows = nb * rows_per_block, warps = ceil_div(rows, per_warp);
        const int cell_threads = ceil_div(ex * nb * s.kp, 32) * 32;
        p.threads = std::min(W_THREADS, std::max(warps * 32, cell_threads));
        if (chunks && (warps * 32 > W_THREADS || pitch > chunks * 128)) continue;
        p.smem = walk_floats(ex, chunks > 0, rows, pitch) * sizeof(float);
        if (p.smem > W_SMEM_MAX || cell_threads > W_THREADS) continue;
        // CTAs of an SM: by the registers (128 a thread) and the shared memory.
        const int per_sm = std::max(1, std::min(W_THREADS / (ceil_div(p.threads, 128) * 128), (int)(W_SMEM_MAX / (p.smem + 1024))));
        const long long groups = ((long long)s.rows + ex - 1) / ex, one_each = walk_clusters(ctx, cs);
        const long long rounds = (groups + one_each * per_sm - 1) / (one_each * per_sm);
        const double share = (double)std::min<long long>(per_sm, (groups + one_each - 1) / one_each);
        const int pieces = pitch / 128, passes = ceil_div(warps, p.threads / 32);
        double cycles = 2500.0 + (cs > 1 ? 310.0 : 0.0) + 115.0 * passes * pieces * ex +
                        5.6 * share * ceil_div(warps, 4) * per_warp * ex;
        if (!chunks) cycles += 10.6 * share * rows * pieces + ((ex >= 4 ? 80.0 : 0.0) + (ex == 8 ? 325.0 : 0.0)) * passes * pieces;
        if (form_dense(form)) cycles += 385.0 + (135.0 + 70.0 * ex) * pieces;
        p.us = 3.0 + (double)rounds * s.T * cycles / 1900.0;
        if (p.us < best.us) best = p;
      }
  return best;
}

template <int EX, int FORM, class Walk>
dlb_status launch_walk(dlb_ctx *ctx, const Walk &walk, const WalkPlan &p) {
  if constexpr (form_exists(FORM, EX)) {
    auto kernel = walk_kernel<EX, FORM>(walk);
    static bool ready[MAX_DEVICES] = {};
    if (!ready[ctx->device]) {
      DLB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)W_SMEM_MAX));
      ready[ctx->device] = true;
    }
    const unsigned grid = (unsigned)(ceil_div(walk.s.rows, EX) * p.cs);
    if (p.cs == 1) {
      DLB_LAUNCH_KERNEL(ctx, kernel, grid, p.threads, p.smem, walk);
    } else {
      DLB_CUDA(launch_kernel_cluster(ctx, kernel, dim3(grid), dim3(p.threads), p.smem, (unsigned)p.cs, walk));
    }
    DLB_LAUNCHED(ctx);
  }
  return DLB_OK;
}
template <int FORM, class Walk>
dlb_status launch_walk(dlb_ctx *ctx, const Walk &walk, const WalkPlan &p) {
  switch (p.ex) {
    case 1: return launch_walk<1, FORM>(ctx, walk, p);
    case 2: return launch_walk<2, FORM>(ctx, walk, p);
    case 4: return launch_walk<4, FORM>(ctx, walk, p);
    case 5: return launch_walk<5, FORM>(ctx, walk, p);
  }
  return launch_walk<8, FORM>(ctx, walk, p);
}
template <int FORM, class Walk>
dlb_status launch_form(dlb_ctx *ctx, const Walk &walk, const WalkPlan &p) {
  if constexpr (FORM + 1 < W_NUM_FORMS)
    if (p.form != FORM) return launch_form<FORM + 1>(ctx, walk, p);
  return launch_walk<FORM>(ctx, walk, p);
}
template <class Walk>
dlb_status run_walk(dlb_ctx *ctx, Walk walk, const WalkPlan &p) {
  walk.s.cs = p.cs, walk.s.status = ctx->d_status;
  return launch_form<0>(ctx, walk, p);
}

WalkShape walk_shape(int rows, int T, int blocks, int cells) {
  int kp = 1;
  while (kp < cells) kp *= 2;
  return {rows, T, blocks, cells, kp, 1, nullptr};
}

// A step on its own: its product, and a launch of the cells' kernel.
double step_by_step_us(const dlb_ctx *ctx, const WalkShape &s, int N, int K) {
  return (double)s.T * (std::min(gemm_small_us(ctx, s.rows, N, K), gemm_direct_us(ctx, s.rows, N, K)) + 5.0);
}

}  // namespace

dlb_status lstm_forward_walk(dlb_ctx *ctx, const float *g_in, const float *w_rec, const float *bias, const float *peep,
                             float *z, float *c, float *ca, float *h, float *gi, float *gf, float *go, int rows, int T,
                             int blocks, int cells, bool *done) {
  const WalkShape s = walk_shape(rows, T, blocks, cells);
  const int C = blocks * cells, G = C + 3 * blocks;
  const WalkPlan p = plan_walk(ctx, s, cells + 3, pad128(C));
  *done = p.us < step_by_step_us(ctx, s, G, C);
  if (!*done) return DLB_OK;
  return run_walk(ctx, ForwardWalk{s, g_in, w_rec, bias, peep, z, c, ca, h, gi, gf, go}, p);
}

dlb_status lstm_backward_walk(dlb_ctx *ctx, float *dH, const float *w_rec, const float *z, const float *ca,
                              const float *c, const float *gi, const float *gf, const float *go, const float *peep,
                              float *d, int rows, int T, int blocks, int cells, bool *done) {
  const WalkShape s = walk_shape(rows, T, blocks, cells);
  const int C = blocks * cells, G = C + 3 * blocks;
  const WalkPlan p = plan_walk(ctx, s, cells, error_pitch(blocks, cells));
  *done = p.us < step_by_step_us(ctx, s, C, G);
  if (!*done) return DLB_OK;
  return run_walk(ctx, BackwardWalk{s, dH, w_rec, z, ca, c, gi, gf, go, peep, d}, p);
}

}  // namespace dlb
