// LSTM / GRU over a whole sequence in one launch per direction.
//
// The recurrence is a serial chain of T small products: launched step by step (hidden projection, gates, and their
// backward) a step of batch 32, hidden 256 took 210 us, nearly all of it launches and half-empty kernels.  Here the
// batch is cut into slices of BS rows, which do not interact, and each slice is one thread-block cluster (1, 2, 4 or 8
// CTAs).  CTA r of a cluster owns the gates of hidden units [r Hs, (r + 1) Hs): its part of the recurrent matrix stays
// on the SM as fp32 for all steps (in registers, else in shared memory; what does not fit there either is read from L2
// at every step).  The new hidden values (or gate gradients) go straight into the shared memory of every CTA of the
// cluster (st.async); each CTA waits on its own mbarrier for the bytes of a step, and two alternating buffers are
// enough because nobody can run a step ahead of the slowest.  Arithmetic is fp32 multiply-adds as in the step-by-step
// kernels.
//
// A step is bound by latency: the product, two block barriers, the gates and the way to the other CTAs; everything a step
// needs from global memory is fetched one step ahead.  How many clusters of eight are on the chip at once is asked of the
// driver (it is fewer than SMs / 8, a cluster lies within one part of the chip): LSTM 256, batch 32, 64 steps ran as 16
// clusters of which not all fitted, 270 us forward and 301 backward for two waves of 150 and 180; on 8 clusters 134 and
// 149, on 11 (slices of three rows) 121 and 134 (GRU: 157 and 179 -> 122 and 123).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "../common/ptx.cuh"
#include "../common/status.h"
#include "../include/ferrum_kernels.h"

namespace fb {
namespace {

namespace cg = cooperative_groups;

constexpr int kT = 512;  // threads

__device__ __forceinline__ float sigm(float x) { return 1.f / (1.f + expf(-x)); }

__device__ __forceinline__ void cp_async4(float* smem_dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(ptx::smem_u32(smem_dst)), "l"(src) : "memory");
}

struct SeqArgs {
  const float *xi, *w, *bias, *h0, *c0;   // xi [T, B, G H]; w [K, ...] as the direction reads it; bias [G H] or NULL
  float *hs, *hs_kept, *cs, *saved, *c_last;  // [T, B, H], the same and [T, B, H], [T, B, 4 H] (NULL: not kept), [B, H]
  const float *d_hs, *d_c_last, *hs_in, *cs_in, *saved_in;  // backward inputs (d_* may be NULL)
  float *dxi, *dhh, *dh0, *dc0;           // [T, B, G H], GRU: the hidden side's gradient, [B, H], [B, H] (NULL)
  int T, B, H, hs_units, rows4, k_res;
  int32_t* status;
  unsigned long long timeout_ns;
};

// How a CTA's threads share the product of its `rows4` rows (a multiple of 4) with a vector v[k][BS] of K entries: a thread
// takes four rows and a slice of k, the `ks_n` partial sums of an output meet in part[ks][b][row].
constexpr int piece_k(int bs) { return bs == 3 ? 4 : 4 / bs; }    // weights in registers: k of a piece of the vector,
constexpr int piece_vec(int bs) { return bs == 3 ? 3 : 1; }        // its 16-byte parts
struct Tile {
  int quads, ks_n;        // row quads, slices
  int pieces;             // weights in registers: pieces of the vector per slice
  int threads, pitch;     // threads that add an output's slices (a power of two within a warp), floats per slice of part
  __host__ __device__ int vec(int K, int bs, bool reg) const {
    return reg ? ks_n * pieces * piece_vec(bs) * 4 : (K + 3) / 4 * 4 * bs;
  }
};
__host__ __device__ inline Tile tile_of(int rows4, int K, int bs, bool reg) {
  Tile t;
  t.quads = rows4 / 4;
  t.ks_n = kT / t.quads;
  const int all = bs == 3 ? (K + 3) / 4 : (K * bs + 3) / 4;
  if (reg && t.ks_n > all) t.ks_n = all;
  t.pieces = (all + t.ks_n - 1) / t.ks_n;
  const int n = rows4 * bs;
  t.threads = 1;
  while (t.threads < 32 && t.threads * 2 * n <= kT) t.threads *= 2;
  // the threads of an output read different slices: shifted so that a warp's reads fall into different banks (not where
  // the weights want the shared memory)
  t.pitch = n + (!reg || t.threads == 1 ? 0 : t.threads >= 8 ? 4 : 32 / t.threads);
  return t;
}

// Weights from shared memory or, past k_res, from L2.  Threads are (k slice, row quad); lanes of a warp read the quads of
// one k: conflict-free.
template <int BS, class Stream>
__device__ __forceinline__ void matvec(const float* wsm, int k_res, int K, int rows4, int pitch, const float* v, float* part,
                                       Stream stream_w) {
  const int rq_n = rows4 >> 2, ks_n = kT / rq_n;
  const int ks = threadIdx.x / rq_n, rq = threadIdx.x - ks * rq_n;
  if (ks >= ks_n) return;
  float acc[4][BS];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int b = 0; b < BS; ++b) acc[i][b] = 0.f;
  int k = ks;
#pragma unroll 4
  for (; k < k_res; k += ks_n) {
    const float4 w = *reinterpret_cast<const float4*>(wsm + k * rows4 + rq * 4);
    float x[BS];
#pragma unroll
    for (int b = 0; b < BS; ++b) x[b] = v[k * BS + b];
#pragma unroll
    for (int b = 0; b < BS; ++b) {
      acc[0][b] = fmaf(w.x, x[b], acc[0][b]);
      acc[1][b] = fmaf(w.y, x[b], acc[1][b]);
      acc[2][b] = fmaf(w.z, x[b], acc[2][b]);
      acc[3][b] = fmaf(w.w, x[b], acc[3][b]);
    }
  }
#pragma unroll 4
  for (; k < K; k += ks_n) {
    float w[4];
    stream_w(k, rq * 4, w);
#pragma unroll
    for (int b = 0; b < BS; ++b) {
      const float x = v[k * BS + b];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i][b] = fmaf(w[i], x, acc[i][b]);
    }
  }
  float* p = part + ks * pitch + rq * 4;
#pragma unroll
  for (int b = 0; b < BS; ++b)
    *reinterpret_cast<float4*>(p + b * rows4) = make_float4(acc[0][b], acc[1][b], acc[2][b], acc[3][b]);
}

// The same product with the weights in registers: four rows and up to kKpt k per thread.  What a step then moves is the
// vector, and a 16-byte read takes four cycles of the shared memory's 128 bytes per cycle even where all lanes read the
// same address: with two rows and 32 k per thread that was 1470 cycles at LSTM 256 on 8 CTAs, two batch rows.  Slice ks
// takes the pieces ks, ks + ks_n, ... (16 bytes each, 48 for three batch rows): neighbouring slices in a warp read
// neighbouring pieces.  The multiply-adds take as many cycles as those reads (1024 each of a step's 4180 at LSTM 256 with
// four batch rows; two in one instruction run at half the rate), so a slice is no taller than the chip's clusters make it:
// batch 32 in slices of three on 11 clusters, not of four on eight.
constexpr int kKpt = 16;
template <int BS>
__device__ __forceinline__ void matvec_reg(const float (&w)[4][kKpt], const Tile& t, int rows4, int ks, int rq, const float* v,
                                           float* part) {
  if (ks >= t.ks_n) return;
  constexpr int kPer = piece_k(BS), kVec = piece_vec(BS);
  float acc[4][BS];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int b = 0; b < BS; ++b) acc[i][b] = 0.f;
  const float4* x = reinterpret_cast<const float4*>(v) + ks * kVec;
  auto piece = [&](int j) {
    float e[kVec * 4];
#pragma unroll
    for (int q = 0; q < kVec; ++q) {
      const float4 f = x[j * t.ks_n * kVec + q];
      e[q * 4] = f.x; e[q * 4 + 1] = f.y; e[q * 4 + 2] = f.z; e[q * 4 + 3] = f.w;
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k)
#pragma unroll
      for (int b = 0; b < BS; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][b] = fmaf(w[i][j * kPer + k], e[k * BS + b], acc[i][b]);
  };
  if (t.pieces == kKpt / kPer) {
#pragma unroll
    for (int j = 0; j < kKpt / kPer; ++j) piece(j);
  } else {
#pragma unroll
    for (int j = 0; j < kKpt / kPer; ++j)
      if (j < t.pieces) piece(j);
  }
  float* p = part + ks * t.pitch + rq * 4;
#pragma unroll
  for (int b = 0; b < BS; ++b)
    *reinterpret_cast<float4*>(p + b * rows4) = make_float4(acc[0][b], acc[1][b], acc[2][b], acc[3][b]);
}
// This thread's weights: at(row) is the address of the row's first one or NULL, `step` the distance from k to k + 1.
template <int BS, class At>
__device__ __forceinline__ void load_weights(float (&w)[4][kKpt], const Tile& t, int K, int ks, int rq, long long step, At at) {
  constexpr int kPer = piece_k(BS);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float* p = ks < t.ks_n ? at(rq * 4 + i) : nullptr;
#pragma unroll
    for (int j = 0; j < kKpt; ++j) {
      const int k = (ks + j / kPer * t.ks_n) * kPer + j % kPer;
      w[i][j] = p != nullptr && j / kPer < t.pieces && k < K ? __ldg(p + k * step) : 0.f;
    }
  }
}

// Sums the k slices of n = rows4 * BS outputs with all threads: `out` is the thread's first output, `passes` how many it
// has, `step` outputs apart, and `leader` tells who hands the sum on.
struct Fold {
  int part, out, step, passes;
  bool leader;
};
__device__ __forceinline__ Fold fold_of(const Tile& t, int n) {
  Fold f;
  f.part = threadIdx.x & (t.threads - 1);
  f.out = threadIdx.x / t.threads;
  f.step = kT / t.threads;
  f.passes = (n + f.step - 1) / f.step;
  f.leader = f.part == 0;
  return f;
}
// kUnroll: slices in flight.  Registers are short beside the weights (64 of 128): forward with the weights there takes four
// (LSTM 256, one batch row 96.7 -> 91.5 us; with sixteen two batch rows went from 106 to 112), the others, which have fewer
// values to keep, eight (LSTM 256 backward, two batch rows: 97, with four 101; LSTM 512 forward: 988, with four 1014).
template <int kUnroll>
__device__ __forceinline__ float fold_sum(const Fold& f, const Tile& t, const float* part, int o, int n) {
  float s = 0.f;
  if (o < n) {
    const float* p = part + f.part * t.pitch + o;
    const int step = t.threads * t.pitch;
#pragma unroll kUnroll
    for (int ks = f.part; ks < t.ks_n; ks += t.threads, p += step) s += *p;
  }
  for (int d = t.threads >> 1; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  return s;
}

// Values for the same place in the shared memory of every CTA of the cluster; the receivers' mbarriers count the bytes.  A
// thread holds element threadIdx.x of the CTA's `count`, consecutive floats of a vector.  Four travel in a message,
// collected from the warp's lanes, which take the (quad, CTA) pairs in turn; where quads do not lie on 16-byte
// boundaries every thread sends its own value to everybody.
struct Outbox {
  uint32_t first, bar;              // element 0 and the barrier, here
  uint32_t to[2], to_bar[2];        // quads: where this lane's one or two messages go (0: nowhere)
  int count, ncl;
  bool quads, mine;                 // `mine`: this warp sends
};
__device__ __forceinline__ uint32_t at_rank(uint32_t local, int rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  return a;
}
template <int BS>
__device__ __forceinline__ Outbox outbox(float* vec, uint64_t* bar, int u0, int Hs, int H, int ncl) {
  Outbox o;
  o.first = ptx::smem_u32(vec) + u0 * BS * 4;
  o.bar = ptx::smem_u32(bar);
  o.count = max(0, min(Hs, H - u0)) * BS;
  o.ncl = ncl;
  o.quads = Hs * BS % 4 == 0 && H * BS % 4 == 0;
  const int lane = threadIdx.x & 31, e0 = threadIdx.x - lane, q = (lane & 7) * 4;
  o.mine = e0 < o.count;
#pragma unroll
  for (int i = 0; i < 2; ++i) {  // eight quads to up to eight CTAs: one or two rounds of 32 lanes
    const int r = i * 4 + (lane >> 3);
    const bool any = o.quads && r < ncl && e0 + q < o.count;
    o.to[i] = any ? at_rank(o.first + (e0 + q) * 4, r) : 0;
    o.to_bar[i] = any ? at_rank(o.bar, r) : 0;
  }
  return o;
}
// Called by the warps that send, whole.  `offset`: bytes from the vector to the one that is written, `bar`: 0 or 1.
__device__ __forceinline__ void send_all(const Outbox& o, uint32_t offset, int bar, float v) {
  if (!o.quads) {
    const int e = threadIdx.x;
    if (e < o.count)
      for (int r = 0; r < o.ncl; ++r)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(
                         at_rank(o.first + offset + e * 4, r)),
                     "r"(__float_as_uint(v)), "r"(at_rank(o.bar + bar * 8, r))
                     : "memory");
    return;
  }
  const int q = (threadIdx.x & 7) * 4;
  const float a = __shfl_sync(0xffffffffu, v, q), b = __shfl_sync(0xffffffffu, v, q + 1);
  const float c = __shfl_sync(0xffffffffu, v, q + 2), d = __shfl_sync(0xffffffffu, v, q + 3);
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (o.to[i] != 0)
      asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                       o.to[i] + offset),
                   "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(__float_as_uint(d)),
                   "r"(o.to_bar[i] + bar * 8)
                   : "memory");
}

// G = 4: LSTM (input, forget, cell, output); G = 3: GRU (reset, update, new).
template <int G, int BS, bool kReg>
__global__ void __launch_bounds__(kT, 1) seq_fwd_kernel(const SeqArgs a) {
  extern __shared__ __align__(16) float sm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int ncl = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int H = a.H, Hs = a.hs_units, R4 = a.rows4, u0 = rank * Hs, b0 = static_cast<int>(blockIdx.x / ncl) * BS;
  const int nb = min(BS, a.B - b0), GH = G * H;
  __shared__ uint64_t arrived[2];           // hidden values of a step complete, one barrier per buffer
  __shared__ int abort_flag;
  float* wsm = sm;                          // [k_res][R4]
  const Tile tile = tile_of(R4, H, BS, kReg);
  const int n_out = R4 * BS, vec = tile.vec(H, BS, kReg);
  float* hbuf = wsm + a.k_res * R4;         // [2][H][BS], padded
  float* part = hbuf + 2 * vec;             // [slice][b][R4]
  float* pre = part + tile.ks_n * tile.pitch;  // [b][R4]: gate values (GRU's new gate: the hidden projection)
  const int ks = threadIdx.x / tile.quads, rq = threadIdx.x - ks * tile.quads;

  auto weight = [&](int k, int r) {         // a.w = transposed matrix [H][G H]
    const int gate = r / Hs, u = u0 + r - gate * Hs;
    return gate < G && u < H ? __ldg(a.w + static_cast<long long>(k) * GH + gate * H + u) : 0.f;
  };
  for (int i = threadIdx.x; i < a.k_res * R4; i += kT) {
    const int k = i / R4;
    wsm[i] = weight(k, i - k * R4);
  }
  float wreg[4][kKpt];
  if constexpr (kReg)
    load_weights<BS>(wreg, tile, H, ks, rq, GH, [&](int r) {
      const int gate = r / Hs, u = u0 + r - gate * Hs;
      return gate < G && u < H ? a.w + gate * H + u : nullptr;
    });
  for (int i = threadIdx.x; i < 2 * vec; i += kT) {
    const int k = i / BS, b = i - k * BS;
    hbuf[i] = (a.h0 != nullptr && b < nb && k < H) ? a.h0[static_cast<long long>(b0 + b) * H + k] : 0.f;
  }
  // thread <-> (unit, batch row) of the pointwise part
  const int pu = threadIdx.x / BS, pb = threadIdx.x % BS;
  const bool mine = pb < nb && pu < Hs && u0 + pu < H;
  const int unit = u0 + pu;
  const long long row = b0 + pb;
  float c = 0.f;
  if (G == 4 && mine && a.c0 != nullptr) c = a.c0[row * H + unit];
  // the gates' inputs of a step: fetched one step ahead into two alternating buffers.  What a thread folds, adds and
  // fetches is the same at every step: output `o` = (batch row b, row r), worked out once where one pass covers all.
  float* xbuf = pre + n_out;                // [2][b][R4]
  const Fold fd = fold_of(tile, n_out);
  auto place = [&](int o, int& gate, int& u, int& b) {
    b = o / R4;
    const int r = o - b * R4;
    gate = r / Hs;
    u = u0 + r - gate * Hs;
    return o < n_out && b < nb && gate < G && u < H;
  };
  int gate0, uu0, bb0;
  const bool valid0 = place(fd.out, gate0, uu0, bb0);
  const float bias0 = valid0 && a.bias != nullptr ? a.bias[gate0 * H + uu0] : 0.f;
  const float* x0 = a.xi + (valid0 ? static_cast<long long>(b0 + bb0) * GH + gate0 * H + uu0 : 0);
  const long long x_step = static_cast<long long>(a.B) * GH;
  auto fetch_x = [&](int t) {
    if (t >= a.T || !fd.leader) return;
    float* dst = xbuf + (t & 1) * n_out;
    if (valid0) cp_async4(dst + fd.out, x0 + t * x_step);
    for (int o = fd.out + fd.step; o < n_out; o += fd.step) {
      int gate, u, b;
      if (place(o, gate, u, b)) cp_async4(dst + o, a.xi + t * x_step + static_cast<long long>(b0 + b) * GH + gate * H + u);
    }
  };
  const uint32_t bytes = static_cast<uint32_t>(H * BS * 4);  // what a CTA receives per step, its own part included
  if (threadIdx.x == 0) {
    abort_flag = 0;
    ptx::mbar_init(&arrived[0], 1);
    ptx::mbar_init(&arrived[1], 1);
    ptx::fence_mbar_init();
    ptx::mbar_arrive_expect_tx(&arrived[0], bytes);
    ptx::mbar_arrive_expect_tx(&arrived[1], bytes);
  }
  fetch_x(0);
  const long long e_step = static_cast<long long>(a.B) * H;
  const long long e_mine = row * H + unit, e4_mine = row * 4 * H + unit;
  const Outbox box = outbox<BS>(hbuf, arrived, u0, Hs, H, ncl);
  cluster.sync();

  for (int t = 0; t < a.T; ++t) {
    const int buf = t & 1;
    const float* cur = hbuf + buf * vec;
    const float* x = xbuf + buf * n_out;
    if (t > 0) {
      // a wait that gives up (reported) goes on with what is there, so that every thread keeps meeting the same barriers
      if (!ptx::mbar_wait(&arrived[buf], ((t - 1) >> 1) & 1, &abort_flag, a.timeout_ns))
        report_status(a.status, kStatusGemmTimeout, 81, blockIdx.x, t);
      if (threadIdx.x == 0) ptx::mbar_arrive_expect_tx(&arrived[buf], bytes);  // for the step after next
    }
    if constexpr (kReg)
      matvec_reg<BS>(wreg, tile, R4, ks, rq, cur, part);
    else
      matvec<BS>(wsm, a.k_res, H, R4, tile.pitch, cur, part, [&](int k, int r, float (&w)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = weight(k, r + i);
      });
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // gate activations in the threads that add the slices: the serial part below is the cell update alone
    for (int pass = 0, o = fd.out; pass < fd.passes; ++pass, o += fd.step) {
      float s = fold_sum<kReg ? 4 : 8>(fd, tile, part, o, n_out);
      if (!fd.leader || o >= n_out) continue;
      int gate = gate0, u = uu0, b = bb0;
      bool ok = valid0;
      float bias = bias0;
      if (o != fd.out) {
        ok = place(o, gate, u, b);
        bias = ok && a.bias != nullptr ? __ldg(a.bias + gate * H + u) : 0.f;
      }
      if (!ok) continue;
      s += bias;
      if (G == 4) s = gate == 2 ? tanhf(x[o] + s) : sigm(x[o] + s);
      else if (gate < 2) s = sigm(x[o] + s);
      pre[o] = s;
    }
    __syncthreads();
    float h = 0.f, p[G];
    if (mine) {
#pragma unroll
      for (int q = 0; q < G; ++q) p[q] = pre[pb * R4 + q * Hs + pu];
      if constexpr (G == 4) {
        c = p[1] * c + p[0] * p[2];
        h = p[3] * tanhf(c);
      } else {
        const float n = tanhf(x[pb * R4 + 2 * Hs + pu] + p[0] * p[2]);
        h = (1.f - p[1]) * n + p[1] * cur[unit * BS + pb];
        if (a.saved != nullptr) a.saved[e4_mine + 4 * t * e_step + 2 * H] = n;
      }
    }
    if (box.mine && t + 1 < a.T) send_all(box, (buf ^ 1) * vec * 4, buf ^ 1, h);
    if (mine) {  // what the others do not wait for
      a.hs[e_mine + t * e_step] = h;
      if (a.hs_kept != nullptr) a.hs_kept[e_mine + t * e_step] = h;
      if (G == 4 && a.cs != nullptr) a.cs[e_mine + t * e_step] = c;
      if (a.saved != nullptr) {
        float* sv = a.saved + e4_mine + 4 * t * e_step;
        sv[0] = p[0];
        sv[H] = p[1];
        if (G == 4) sv[2 * H] = p[2];
        sv[3 * H] = p[G - 1];
      }
    }
    fetch_x(t + 1);
  }
  if (G == 4 && mine && a.c_last != nullptr) a.c_last[row * H + unit] = c;
  cluster.sync();  // the other CTAs may still write into this one's shared memory
}

template <int G, int BS, bool kReg>
__global__ void __launch_bounds__(kT, 1) seq_bwd_kernel(const SeqArgs a) {
  extern __shared__ __align__(16) float sm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int ncl = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int H = a.H, Hs = a.hs_units, R4 = a.rows4, u0 = rank * Hs, b0 = static_cast<int>(blockIdx.x / ncl) * BS;
  const int nb = min(BS, a.B - b0), K = G * H;
  __shared__ uint64_t arrived[2];           // gate gradients of a step complete, one barrier per buffer
  __shared__ int abort_flag;
  float* wsm = sm;                          // [k_res][R4]: rows of the recurrent matrix, this CTA's columns
  const Tile tile = tile_of(R4, K, BS, kReg);
  const int n_out = R4 * BS, vec = tile.vec(K, BS, kReg);
  float* dbuf = wsm + a.k_res * R4;         // [2][K][BS], padded: gate gradients of the step, all units
  float* part = dbuf + 2 * vec;             // [slice][b][R4]
  float* dh = part + tile.ks_n * tile.pitch;  // [b][R4]: gradient that arrives from the next step
  const int ks = threadIdx.x / tile.quads, rq = threadIdx.x - ks * tile.quads;

  auto weight = [&](int k, int r) {         // a.w = [G H][H]
    return r < Hs && u0 + r < H ? __ldg(a.w + static_cast<long long>(k) * H + u0 + r) : 0.f;
  };
  for (int i = threadIdx.x; i < a.k_res * R4; i += kT) {
    const int k = i / R4;
    wsm[i] = weight(k, i - k * R4);
  }
  float wreg[4][kKpt];
  if constexpr (kReg)
    load_weights<BS>(wreg, tile, K, ks, rq, H, [&](int r) { return r < Hs && u0 + r < H ? a.w + u0 + r : nullptr; });
  for (int i = threadIdx.x; i < 2 * vec; i += kT) dbuf[i] = 0.f;
  for (int i = threadIdx.x; i < n_out; i += kT) dh[i] = 0.f;

  const int pu = threadIdx.x / BS, pb = threadIdx.x % BS;
  const bool mine = pb < nb && pu < Hs && u0 + pu < H;
  const int unit = u0 + pu;
  const long long row = b0 + pb;
  const Fold fd = fold_of(tile, n_out);
  const long long e_step = static_cast<long long>(a.B) * K, e_mine = row * K + unit;
  const Outbox box = outbox<BS>(dbuf, arrived, u0, Hs, H, ncl);
  float carry = 0.f;                        // LSTM: dc; GRU: dh * z of the step after
  if (G == 4 && mine && a.d_c_last != nullptr) carry = a.d_c_last[row * H + unit];
  // what the pointwise part of step t reads from global memory
  struct In {
    float s[4], prev, c, d;
  };
  auto fetch = [&](int t) {
    In v = {};
    if (!mine || t < 0) return v;
    const long long e = (static_cast<long long>(t) * a.B + row) * H + unit;
    const long long e4 = (static_cast<long long>(t) * a.B + row) * 4 * H + unit;
#pragma unroll
    for (int q = 0; q < 4; ++q) v.s[q] = __ldg(a.saved_in + e4 + q * H);
    const float* prev = G == 4 ? a.cs_in : a.hs_in;
    const float* init = G == 4 ? a.c0 : a.h0;
    if (t > 0) v.prev = __ldg(prev + e - static_cast<long long>(a.B) * H);
    else if (init != nullptr) v.prev = __ldg(init + row * H + unit);
    if (G == 4) v.c = __ldg(a.cs_in + e);
    if (a.d_hs != nullptr) v.d = __ldg(a.d_hs + e);
    return v;
  };
  const uint32_t bytes = static_cast<uint32_t>(K * BS * 4);  // what a CTA receives per step, its own part included
  if (threadIdx.x == 0) {
    abort_flag = 0;
    ptx::mbar_init(&arrived[0], 1);
    ptx::mbar_init(&arrived[1], 1);
    ptx::fence_mbar_init();
    ptx::mbar_arrive_expect_tx(&arrived[0], bytes);
    ptx::mbar_arrive_expect_tx(&arrived[1], bytes);
  }
  In in = fetch(a.T - 1);
  cluster.sync();

  for (int t = a.T - 1; t >= 0; --t) {
    const int buf = t & 1;
    float* cur = dbuf + buf * vec;
    float dx[G], dq[G];
#pragma unroll
    for (int q = 0; q < G; ++q) dq[q] = 0.f;
    if (mine) {
      const float g = in.d + dh[pb * R4 + pu] + (G == 3 ? carry : 0.f);
      if constexpr (G == 4) {
        const float i = in.s[0], f = in.s[1], cc = in.s[2], o = in.s[3];
        const float tc = tanhf(in.c);
        const float gc = carry + g * o * (1.f - tc * tc);
        dx[0] = gc * cc * i * (1.f - i);
        dx[1] = gc * in.prev * f * (1.f - f);
        dx[2] = gc * i * (1.f - cc * cc);
        dx[3] = g * tc * o * (1.f - o);
        carry = gc * f;
#pragma unroll
        for (int q = 0; q < G; ++q) dq[q] = dx[q];
      } else {
        const float r = in.s[0], z = in.s[1], nn = in.s[2], hn = in.s[3];
        const float dn = g * (1.f - z) * (1.f - nn * nn);
        dx[0] = dn * hn * r * (1.f - r);
        dx[1] = g * (in.prev - nn) * z * (1.f - z);
        dx[2] = dn;
        dq[0] = dx[0];
        dq[1] = dx[1];
        dq[2] = dn * r;
        carry = g * z;
      }
    }
    if (box.mine) {
#pragma unroll
      for (int q = 0; q < G; ++q) send_all(box, (buf * vec + q * H * BS) * 4, buf, dq[q]);
    }
    if (mine) {  // what the others do not wait for
      const long long e = e_mine + t * e_step;
#pragma unroll
      for (int q = 0; q < G; ++q) {
        a.dxi[e + q * H] = dx[q];
        if (G == 3) a.dhh[e + q * H] = dq[q];
      }
    }
    in = fetch(t - 1);
    if (!ptx::mbar_wait(&arrived[buf], ((a.T - 1 - t) >> 1) & 1, &abort_flag, a.timeout_ns))
      report_status(a.status, kStatusGemmTimeout, 82, blockIdx.x, t);
    if (threadIdx.x == 0) ptx::mbar_arrive_expect_tx(&arrived[buf], bytes);  // for the step after next
    if constexpr (kReg)
      matvec_reg<BS>(wreg, tile, R4, ks, rq, cur, part);
    else
      matvec<BS>(wsm, a.k_res, K, R4, tile.pitch, cur, part, [&](int k, int r, float (&w)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = weight(k, r + i);
      });
    __syncthreads();
    for (int pass = 0, o = fd.out; pass < fd.passes; ++pass, o += fd.step) {
      const float s = fold_sum<8>(fd, tile, part, o, n_out);
      if (fd.leader && o < n_out) dh[o] = s;
    }
    __syncthreads();
  }
  if (mine) {
    if (a.dh0 != nullptr) a.dh0[row * H + unit] = dh[pb * R4 + pu] + (G == 3 ? carry : 0.f);
    if (G == 4 && a.dc0 != nullptr) a.dc0[row * H + unit] = carry;
  }
  cluster.sync();  // the other CTAs may still write into this one's shared memory
}

int smem_limit() {
  static int v = 0;
  if (v == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  }
  return v;
}

struct Plan {
  int ncl, bs, hs_units, rows4, k_res;
  bool reg;  // weights in registers
  size_t smem;
};
// Clusters of `ncl` CTAs, one CTA per SM, that are on the chip at once.
int cluster_slots(int ncl);

// Cluster size: one CTA per 32 hidden units up to eight (a CTA's share of the weights is then what a step has to
// stream from shared memory).  Batch slice: as small as keeps every cluster on the chip at once; three rows only with the
// weights in registers (where shared memory or L2 holds them a step costs what it reads of them, whatever the slice).
bool plan(int G, int B, int H, bool backward, Plan* p) {
  if (H < 1 || H > 1024) return false;
  p->ncl = H >= 256 ? 8 : (H >= 128 ? 4 : (H >= 64 ? 2 : 1));
  const int slots = cluster_slots(p->ncl);
  p->bs = B <= slots ? 1 : (B <= 2 * slots ? 2 : (B <= 3 * slots ? 3 : (B <= 4 * slots ? 4 : 8)));
  p->hs_units = (H + p->ncl - 1) / p->ncl;
  const int rows = backward ? p->hs_units : G * p->hs_units, K = backward ? G * H : H;
  p->rows4 = (rows + 3) / 4 * 4;
  if (p->rows4 / 4 > kT) return false;
  const size_t limit = static_cast<size_t>(smem_limit()) - 1024;
  auto in_registers = [&] { return p->bs <= 4 && tile_of(p->rows4, K, p->bs, true).pieces * piece_k(p->bs) <= kKpt; };
  if (p->bs == 3 && !in_registers()) p->bs = 4;
  for (; p->bs >= 1; p->bs = p->bs == 3 ? 2 : p->bs >> 1) {  // a smaller slice leaves more shared memory to the weights
    p->reg = in_registers();
    const Tile t = tile_of(p->rows4, K, p->bs, p->reg);
    // two vectors, the partial sums, and the gates with their two input buffers
    const size_t fixed = (2 * static_cast<size_t>(t.vec(K, p->bs, p->reg)) + static_cast<size_t>(t.ks_n) * t.pitch +
                          3 * static_cast<size_t>(p->rows4) * p->bs) * 4;
    if (p->hs_units * p->bs > kT || fixed > limit) continue;
    if (p->reg) {
      p->k_res = 0;
      p->smem = fixed;
      return true;
    }
    size_t k = (limit - fixed) / (static_cast<size_t>(p->rows4) * 4);
    if (k > static_cast<size_t>(K)) k = K;
    // streaming up to three quarters of the weights from L2 at every step (3 us at hidden 512) still beats a step of
    // separate launches; beyond that the products are large enough for those
    if (4 * k < static_cast<size_t>(K)) continue;
    p->k_res = static_cast<int>(k);
    p->smem = fixed + k * p->rows4 * 4;
    return true;
  }
  return false;
}

int cluster_slots(int ncl) {
  static std::atomic<int> known[9];
  int n = known[ncl].load(std::memory_order_relaxed);
  if (n > 0) return n;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ncl);
  cfg.blockDim = dim3(kT);
  cfg.dynamicSmemBytes = 0;  // 512 threads of more than 64 registers: one CTA per SM whatever its shared memory
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ncl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, seq_fwd_kernel<4, 2, true>, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    return 1;
  }
  known[ncl].store(n, std::memory_order_relaxed);
  return n;
}

template <int G, int BS, bool kReg>
int run_one(bool backward, const SeqArgs& a, const Plan& p, cudaStream_t st) {
  auto fn = backward ? seq_bwd_kernel<G, BS, kReg> : seq_fwd_kernel<G, BS, kReg>;
  static int configured[2] = {0, 0};
  if (static_cast<int>(p.smem) > configured[backward]) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(p.smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    configured[backward] = static_cast<int>(p.smem);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((a.B + BS - 1) / BS * p.ncl));
  cfg.blockDim = dim3(kT);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = p.ncl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, fn, a));
}
template <int G, int BS>
int run(bool backward, const SeqArgs& a, const Plan& p, cudaStream_t st) {
  if constexpr (BS <= 4) {
    if (p.reg) return run_one<G, BS, true>(backward, a, p, st);
  }
  if constexpr (BS == 3) return -1;  // plan() has three rows with the weights in registers alone
  else return run_one<G, BS, false>(backward, a, p, st);
}
template <int G>
int run_bs(bool backward, const SeqArgs& a, const Plan& p, cudaStream_t st) {
  switch (p.bs) {
    case 1: return run<G, 1>(backward, a, p, st);
    case 2: return run<G, 2>(backward, a, p, st);
    case 3: return run<G, 3>(backward, a, p, st);
    case 4: return run<G, 4>(backward, a, p, st);
    default: return run<G, 8>(backward, a, p, st);
  }
}

}  // namespace
}  // namespace fb

using namespace fb;

extern "C" int fb_rnn_seq_supported(int gates, int B, int H) {
  Plan f, b;
  return (gates == 3 || gates == 4) && B > 0 && plan(gates, B, H, false, &f) && plan(gates, B, H, true, &b);
}

extern "C" int fb_rnn_seq_plan(int gates, int B, int H, int backward) {
  Plan p;
  if ((gates != 3 && gates != 4) || B < 1 || !plan(gates, B, H, backward != 0, &p)) return 0;
  const bool full = p.reg && tile_of(p.rows4, backward ? gates * H : H, p.bs, true).pieces == kKpt / piece_k(p.bs);
  return p.bs + (p.reg ? 16 : 0) + (full ? 32 : 0);
}

extern "C" int fb_rnn_seq_fwd(int gates, const float* xi, const float* w_t, const float* bias, const float* h0,
                              const float* c0, float* hs, float* hs_kept, float* cs, float* saved, float* c_last, int T,
                              int B, int H, int32_t* status, cudaStream_t stream) {
  if (T <= 0 || B <= 0 || H <= 0) return 0;
  Plan p;
  if ((gates != 3 && gates != 4) || !plan(gates, B, H, false, &p)) return -1;
  SeqArgs a = {};
  a.xi = xi; a.w = w_t; a.bias = bias; a.h0 = h0; a.c0 = c0;
  a.hs = hs; a.hs_kept = hs_kept; a.cs = cs; a.saved = saved; a.c_last = c_last;
  a.T = T; a.B = B; a.H = H; a.status = status; a.timeout_ns = 2000000000ull;
  a.hs_units = p.hs_units; a.rows4 = p.rows4; a.k_res = p.k_res;
  return gates == 4 ? run_bs<4>(false, a, p, stream) : run_bs<3>(false, a, p, stream);
}

extern "C" int fb_rnn_seq_bwd(int gates, const float* w, const float* h0, const float* c0, const float* hs,
                              const float* cs, const float* saved, const float* d_hs, const float* d_c_last, float* dxi,
                              float* dhh, float* dh0, float* dc0, int T, int B, int H, int32_t* status,
                              cudaStream_t stream) {
  if (T <= 0 || B <= 0 || H <= 0) return 0;
  Plan p;
  if ((gates != 3 && gates != 4) || !plan(gates, B, H, true, &p) || (gates == 3 && dhh == nullptr)) return -1;
  SeqArgs a = {};
  a.w = w; a.h0 = h0; a.c0 = c0; a.hs_in = hs; a.cs_in = cs; a.saved_in = saved;
  a.d_hs = d_hs; a.d_c_last = d_c_last; a.dxi = dxi; a.dhh = dhh; a.dh0 = dh0; a.dc0 = dc0;
  a.T = T; a.B = B; a.H = H; a.status = status; a.timeout_ns = 2000000000ull;
  a.hs_units = p.hs_units; a.rows4 = p.rows4; a.k_res = p.k_res;
  return gates == 4 ? run_bs<4>(true, a, p, stream) : run_bs<3>(true, a, p, stream);
}
