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
// A step is bound by latency: the product (700 cycles at LSTM 256 on 8 CTAs), two block barriers, the gates and the
// way to the other CTAs; everything a step needs from global memory is fetched one step ahead.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

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

// part[ks][rows4][BS] += over k = ks, ks + KS, ... of w[k][4 rows] * v[k][BS]; then out[r][b] = sum over ks.
// Threads are (row quad, k slice); lanes of a warp read consecutive k (or the quads of one k): conflict-free.
template <int BS, class Stream>
__device__ __forceinline__ void matvec(const float* wsm, int k_res, int K, int rows4, const float* v, float* part,
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
  float* p = part + (ks * rows4 + rq * 4) * BS;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int b = 0; b < BS; ++b) p[i * BS + b] = acc[i][b];
}

// The same product with the weights in registers: a thread owns two rows and kKpt consecutive k, so a step reads only
// the vector (one broadcast per k) from shared memory.  LSTM 256 on 8 CTAs: 2800 -> 700 cycles per step.
constexpr int kKpt = 32;
struct RegTile {
  int pairs, ks_n, kpt;  // row pairs, k slices, k per slice (<= kKpt)
};
__host__ __device__ inline RegTile reg_tile(int rows4, int K) {
  RegTile r;
  r.pairs = rows4 / 2;
  r.ks_n = kT / r.pairs;
  if (r.ks_n > K / 4) r.ks_n = K / 4 > 0 ? K / 4 : 1;
  r.kpt = ((K + r.ks_n - 1) / r.ks_n + 3) / 4 * 4;
  return r;
}
struct RegLane {
  int n, v_at, part_at;  // k of this thread's slice (<= 0: idle), its offsets in the vector and in `part`
};
template <int BS>
__device__ __forceinline__ RegLane reg_lane(const RegTile rt, int K, int rows4) {
  const int ks = threadIdx.x / rt.pairs, rp = threadIdx.x - ks * rt.pairs;
  return RegLane{ks < rt.ks_n ? max(0, min(rt.kpt, K - ks * rt.kpt)) : -1, ks * rt.kpt * BS, (ks * rows4 + rp * 2) * BS};
}
template <int BS>
__device__ __forceinline__ void matvec_reg(const float (&w)[2][kKpt], const RegLane l, const float* v, float* part) {
  if (l.n < 0) return;
  float acc[2][BS];
#pragma unroll
  for (int b = 0; b < BS; ++b) acc[0][b] = acc[1][b] = 0.f;
  const float* x = v + l.v_at;
#pragma unroll
  for (int k0 = 0; k0 < kKpt; k0 += 4) {
    if (k0 < l.n) {  // the vector is padded with zeros to a multiple of four
      float xv[4 * BS];
#pragma unroll
      for (int i = 0; i < BS; ++i) {
        const float4 f = *reinterpret_cast<const float4*>(x + k0 * BS + 4 * i);
        xv[4 * i] = f.x; xv[4 * i + 1] = f.y; xv[4 * i + 2] = f.z; xv[4 * i + 3] = f.w;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int b = 0; b < BS; ++b) {
          acc[0][b] = fmaf(w[0][k0 + k], xv[k * BS + b], acc[0][b]);
          acc[1][b] = fmaf(w[1][k0 + k], xv[k * BS + b], acc[1][b]);
        }
    }
  }
  float* p = part + l.part_at;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int b = 0; b < BS; ++b) p[i * BS + b] = acc[i][b];
}

// Sums the k slices of n = rows4 * BS outputs with all threads: `threads` of them (a power of two within a warp) share
// an output; `out` is the thread's first output and `leader` tells who hands the sum on.
struct Fold {
  int threads, part, out, step;
  bool leader;
};
__device__ __forceinline__ Fold fold_of(int n) {
  Fold f;
  f.threads = 1;
  while (f.threads < 32 && f.threads * 2 * n <= kT) f.threads *= 2;
  f.part = threadIdx.x & (f.threads - 1);
  f.out = threadIdx.x / f.threads;
  f.step = kT / f.threads;
  f.leader = f.part == 0;
  return f;
}
__device__ __forceinline__ float fold_sum(const Fold& f, const float* part, int o, int n, int ks_n) {
  float s = 0.f;
  if (o < n) {
#pragma unroll 8
    for (int ks = f.part; ks < ks_n; ks += f.threads) s += part[ks * n + o];
  }
  for (int d = f.threads >> 1; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  return s;
}

// A value for the same place in the shared memory of every CTA of the cluster; the receivers' mbarriers count the bytes.
__device__ __forceinline__ void send(uint32_t local_addr, uint32_t local_bar, int rank, float v) {
  uint32_t dst, bar;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(local_addr), "r"(rank));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(local_bar), "r"(rank));
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}

// G = 4: LSTM (input, forget, cell, output); G = 3: GRU (reset, update, new).
template <int G, int BS, bool kReg>
__global__ void __launch_bounds__(kT, 1) seq_fwd_kernel(const SeqArgs a) {
  extern __shared__ float sm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int ncl = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int H = a.H, Hs = a.hs_units, R4 = a.rows4, u0 = rank * Hs, b0 = static_cast<int>(blockIdx.x / ncl) * BS;
  const int nb = min(BS, a.B - b0), GH = G * H;
  __shared__ uint64_t arrived[2];           // hidden values of a step complete, one barrier per buffer
  __shared__ int abort_flag;
  float* wsm = sm;                          // [k_res][R4]
  float* hbuf = wsm + a.k_res * R4;         // [2][H][BS]
  const int Hp = (H + 3) / 4 * 4;
  float* part = hbuf + 2 * Hp * BS;         // [4 * kT][BS]
  float* pre = part + 4 * kT * BS;          // [R4][BS]: gate values (GRU's new gate: the hidden projection)
  const RegTile rt = reg_tile(R4, H);
  const RegLane lane = reg_lane<BS>(rt, H, R4);
  const int ks_n = kReg ? rt.ks_n : kT / (R4 >> 2);

  auto weight = [&](int k, int r) {         // a.w = transposed matrix [H][G H]
    const int gate = r / Hs, u = u0 + r - gate * Hs;
    return gate < G && u < H ? __ldg(a.w + static_cast<long long>(k) * GH + gate * H + u) : 0.f;
  };
  for (int i = threadIdx.x; i < a.k_res * R4; i += kT) {
    const int k = i / R4;
    wsm[i] = weight(k, i - k * R4);
  }
  float wreg[2][kKpt];
  if constexpr (kReg) {
    const int ks = threadIdx.x / rt.pairs, rp = threadIdx.x - ks * rt.pairs;
#pragma unroll
    for (int k = 0; k < kKpt; ++k) {
      const int kk = ks * rt.kpt + k;
      const bool in = ks < rt.ks_n && k < rt.kpt && kk < H;
      wreg[0][k] = in ? weight(kk, rp * 2) : 0.f;
      wreg[1][k] = in ? weight(kk, rp * 2 + 1) : 0.f;
    }
  }
  for (int i = threadIdx.x; i < 2 * Hp * BS; i += kT) {
    const int k = i / BS, b = i - k * BS;
    hbuf[i] = (a.h0 != nullptr && b < nb && k < H) ? a.h0[static_cast<long long>(b0 + b) * H + k] : 0.f;
  }
  // thread <-> (unit, batch row) of the pointwise part
  const int pu = threadIdx.x % Hs, pb = threadIdx.x / Hs;
  const bool mine = pb < nb && u0 + pu < H;
  const int unit = u0 + pu;
  const long long row = b0 + pb;
  float c = 0.f;
  if (G == 4 && mine && a.c0 != nullptr) c = a.c0[row * H + unit];
  // the gates' inputs of a step: fetched one step ahead into two alternating buffers.  What a thread folds, adds and
  // fetches is the same at every step: output `o` = (row r, batch row b), worked out once where one pass covers all.
  float* xbuf = pre + R4 * BS;              // [2][R4 * BS]
  const int n_out = R4 * BS;
  const Fold fd = fold_of(n_out);
  auto place = [&](int o, int& gate, int& u, int& b) {
    const int r = o / BS;
    b = o - r * BS;
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
  const uint32_t bytes = static_cast<uint32_t>(H * nb * 4);  // what a CTA receives per step, its own part included
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
  const uint32_t send_at = ptx::smem_u32(hbuf) + (unit * BS + pb) * 4;
  cluster.sync();

  for (int t = 0; t < a.T; ++t) {
    const int buf = t & 1;
    const float* cur = hbuf + buf * Hp * BS;
    const float* x = xbuf + buf * n_out;
    if (t > 0) {
      // a wait that gives up (reported) goes on with what is there, so that every thread keeps meeting the same barriers
      if (!ptx::mbar_wait(&arrived[buf], ((t - 1) >> 1) & 1, &abort_flag, a.timeout_ns))
        report_status(a.status, kStatusGemmTimeout, 81, blockIdx.x, t);
      if (threadIdx.x == 0) ptx::mbar_arrive_expect_tx(&arrived[buf], bytes);  // for the step after next
    }
    if constexpr (kReg)
      matvec_reg<BS>(wreg, lane, cur, part);
    else
      matvec<BS>(wsm, a.k_res, H, R4, cur, part, [&](int k, int r, float (&w)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = weight(k, r + i);
      });
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // gate activations in the threads that add the slices: the serial part below is the cell update alone
    for (int o = fd.out; o < (n_out + fd.step - 1) / fd.step * fd.step; o += fd.step) {
      float s = fold_sum(fd, part, o, n_out, ks_n);
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
      for (int q = 0; q < G; ++q) p[q] = pre[(q * Hs + pu) * BS + pb];
      if constexpr (G == 4) {
        c = p[1] * c + p[0] * p[2];
        h = p[3] * tanhf(c);
      } else {
        const float n = tanhf(x[(2 * Hs + pu) * BS + pb] + p[0] * p[2]);
        h = (1.f - p[1]) * n + p[1] * cur[unit * BS + pb];
        if (a.saved != nullptr) a.saved[e4_mine + 4 * t * e_step + 2 * H] = n;
      }
      if (t + 1 < a.T) {
        const int nxt = buf ^ 1;
        for (int r = 0; r < ncl; ++r)
          send(send_at + nxt * Hp * BS * 4, ptx::smem_u32(&arrived[nxt]), r, h);
      }
      // what the others do not wait for
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
  extern __shared__ float sm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int ncl = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int H = a.H, Hs = a.hs_units, R4 = a.rows4, u0 = rank * Hs, b0 = static_cast<int>(blockIdx.x / ncl) * BS;
  const int nb = min(BS, a.B - b0), K = G * H;
  __shared__ uint64_t arrived[2];           // gate gradients of a step complete, one barrier per buffer
  __shared__ int abort_flag;
  float* wsm = sm;                          // [k_res][R4]: rows of the recurrent matrix, this CTA's columns
  float* dbuf = wsm + a.k_res * R4;         // [2][K][BS]: gate gradients of the step, all units
  const int Kp = (K + 3) / 4 * 4;
  float* part = dbuf + 2 * Kp * BS;         // [4 * kT][BS]
  float* dh = part + 4 * kT * BS;           // [R4][BS]: gradient that arrives from the next step
  const RegTile rt = reg_tile(R4, K);
  const RegLane lane = reg_lane<BS>(rt, K, R4);
  const int ks_n = kReg ? rt.ks_n : kT / (R4 >> 2);

  auto weight = [&](int k, int r) {         // a.w = [G H][H]
    return r < Hs && u0 + r < H ? __ldg(a.w + static_cast<long long>(k) * H + u0 + r) : 0.f;
  };
  for (int i = threadIdx.x; i < a.k_res * R4; i += kT) {
    const int k = i / R4;
    wsm[i] = weight(k, i - k * R4);
  }
  float wreg[2][kKpt];
  if constexpr (kReg) {
    const int ks = threadIdx.x / rt.pairs, rp = threadIdx.x - ks * rt.pairs;
#pragma unroll
    for (int k = 0; k < kKpt; ++k) {
      const int kk = ks * rt.kpt + k;
      const bool in = ks < rt.ks_n && k < rt.kpt && kk < K;
      wreg[0][k] = in ? weight(kk, rp * 2) : 0.f;
      wreg[1][k] = in ? weight(kk, rp * 2 + 1) : 0.f;
    }
  }
  for (int i = threadIdx.x; i < 2 * Kp * BS; i += kT) dbuf[i] = 0.f;
  for (int i = threadIdx.x; i < R4 * BS; i += kT) dh[i] = 0.f;

  const int pu = threadIdx.x % Hs, pb = threadIdx.x / Hs;
  const bool mine = pb < nb && u0 + pu < H;
  const int unit = u0 + pu;
  const long long row = b0 + pb;
  const int n_out = R4 * BS;
  const Fold fd = fold_of(n_out);
  const long long e_step = static_cast<long long>(a.B) * K, e_mine = row * K + unit;
  const uint32_t send_at = ptx::smem_u32(dbuf) + (unit * BS + pb) * 4;
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
  const uint32_t bytes = static_cast<uint32_t>(K * nb * 4);  // what a CTA receives per step, its own part included
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
    float* cur = dbuf + buf * Kp * BS;
    float dx[G], dq[G];
    if (mine) {
      const float g = in.d + dh[pu * BS + pb] + (G == 3 ? carry : 0.f);
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
      for (int r = 0; r < ncl; ++r) {
#pragma unroll
        for (int q = 0; q < G; ++q)
          send(send_at + (buf * Kp + q * H) * BS * 4, ptx::smem_u32(&arrived[buf]), r, dq[q]);
      }
      // what the others do not wait for
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
      matvec_reg<BS>(wreg, lane, cur, part);
    else
      matvec<BS>(wsm, a.k_res, K, R4, cur, part, [&](int k, int r, float (&w)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = weight(k, r + i);
      });
    __syncthreads();
    for (int o = fd.out; o < (n_out + fd.step - 1) / fd.step * fd.step; o += fd.step) {
      const float s = fold_sum(fd, part, o, n_out, ks_n);
      if (fd.leader && o < n_out) dh[o] = s;
    }
    __syncthreads();
  }
  if (mine) {
    if (a.dh0 != nullptr) a.dh0[row * H + unit] = dh[pu * BS + pb] + (G == 3 ? carry : 0.f);
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

int sm_count() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}

struct Plan {
  int ncl, bs, hs_units, rows4, k_res;
  bool reg;  // weights in registers
  size_t smem;
};
// Cluster size: one CTA per 32 hidden units up to eight (a CTA's share of the weights is then what a step has to
// stream from shared memory).  Batch slice: as small as keeps every cluster on the chip at once.
bool plan(int G, int B, int H, bool backward, Plan* p) {
  if (H < 1 || H > 1024) return false;
  p->ncl = H >= 256 ? 8 : (H >= 128 ? 4 : (H >= 64 ? 2 : 1));
  const int slots = sm_count() / p->ncl;
  p->bs = B <= slots ? 1 : (B <= 2 * slots ? 2 : (B <= 4 * slots ? 4 : 8));
  p->hs_units = (H + p->ncl - 1) / p->ncl;
  const int rows = backward ? p->hs_units : G * p->hs_units, K = backward ? G * H : H;
  p->rows4 = (rows + 3) / 4 * 4;
  if (p->rows4 / 4 > kT) return false;
  const size_t limit = static_cast<size_t>(smem_limit()) - 1024;
  for (; p->bs >= 1; p->bs >>= 1) {  // a smaller slice leaves more shared memory to the weights
    const size_t fixed = (2 * static_cast<size_t>((K + 3) / 4 * 4) + 4 * kT + 3 * p->rows4) * p->bs * 4;
    if (p->hs_units * p->bs > kT || fixed > limit) continue;
    p->reg = p->bs <= 4 && reg_tile(p->rows4, K).kpt <= kKpt;
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
  return run_one<G, BS, false>(backward, a, p, st);
}
template <int G>
int run_bs(bool backward, const SeqArgs& a, const Plan& p, cudaStream_t st) {
  switch (p.bs) {
    case 1: return run<G, 1>(backward, a, p, st);
    case 2: return run<G, 2>(backward, a, p, st);
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
