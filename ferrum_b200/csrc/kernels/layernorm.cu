// Per-row LayerNorm forward / backward, optionally fused with a preceding GELU
// (the Linear -> GELU -> LayerNorm block reads the pre-activation once and
// writes the normalised output once; the backward produces the gradient of the
// pre-activation plus the three column reductions d_gamma, d_beta and the
// column sum of dx, which is the bias gradient of the preceding Linear).
//
// Reference: ferrum-nn/src/norm.rs:13-68,226-239 (module + functional; the
// reference normalises with the statistics of the whole tensor — this kernel
// normalises each row of `normalized_shape`, like the row-wise variant at
// ferrum-nn/src/transformer.rs:316-342) and ferrum-nn/src/activation.rs:254-262 (GELU).
//
// Fast path: a row lives in registers (TPR threads x K vectors of 8 elements, 16-byte
// accesses), two-pass mean / variance on registers, column partials accumulate in
// registers across the rows a block owns and are written once to
// partial[nblk][3][cols]; a second kernel folds the partials.  Register budgets are
// kept small enough for two to four 256-thread blocks per SM: these kernels are
// bandwidth-bound and need the bytes in flight.
// Rows of odd width or address: a row lives in registers there, too, element by
// element (ln_*_any_kernel), or is re-read, with column sums by atomicAdd
// (ln_*_generic), whichever is faster for its size; see any_fwd and any_bwd.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdlib>

#include "../common/ptx.cuh"
#include "../common/status.h"
#include "../include/ferrum_kernels.h"

namespace fb {
namespace {

constexpr float kGeluC = 0.7978845608028654f;
constexpr float kGeluA = 0.044715f;

// FAST = hardware tanh.approx (bf16 data: its 2^-11 error is below the storage rounding);
// otherwise the accurate tanhf (fp32 parity path).
template <bool FAST>
__device__ __forceinline__ float tanh_sel(float u) {
  if (FAST) {
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
    return t;
  }
  return tanhf(u);
}
template <bool FAST>
__device__ __forceinline__ float gelu_f(float x) {
  return 0.5f * x * (1.f + tanh_sel<FAST>(kGeluC * (x + kGeluA * x * x * x)));
}
// value and derivative from one tanh
template <bool FAST>
__device__ __forceinline__ void gelu_both(float x, float& val, float& der) {
  const float t = tanh_sel<FAST>(kGeluC * (x + kGeluA * x * x * x));
  val = 0.5f * x * (1.f + t);
  der = 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * kGeluC * (1.f + 3.f * kGeluA * x * x);
}

// Eight consecutive elements: one 16-byte access for bf16, two for fp32.
template <typename T>
struct V8;
template <>
struct V8<float> {
  static constexpr bool kFastMath = false;
  struct Raw { float4 a, b; };
  static __device__ __forceinline__ Raw ld(const float* p) {
    Raw r;
    r.a = *reinterpret_cast<const float4*>(p);
    r.b = *reinterpret_cast<const float4*>(p + 4);
    return r;
  }
  static __device__ __forceinline__ void unpack(const Raw& r, float (&f)[8]) {
    f[0] = r.a.x; f[1] = r.a.y; f[2] = r.a.z; f[3] = r.a.w; f[4] = r.b.x; f[5] = r.b.y; f[6] = r.b.z; f[7] = r.b.w;
  }
  static __device__ __forceinline__ void st(float* p, const float (&f)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(f[4], f[5], f[6], f[7]);
  }
  static __device__ __forceinline__ float ld1(const float* p) { return *p; }
  static __device__ __forceinline__ void st1(float* p, float v) { *p = v; }
};
template <>
struct V8<__nv_bfloat16> {
  static constexpr bool kFastMath = true;
  using Raw = uint4;
  static __device__ __forceinline__ Raw ld(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
  static __device__ __forceinline__ void unpack(const Raw& r, float (&f)[8]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 t = __bfloat1622float2(h[i]);
      f[2 * i] = t.x;
      f[2 * i + 1] = t.y;
    }
  }
  static __device__ __forceinline__ void st(__nv_bfloat16* p, const float (&f)[8]) {
    uint4 u;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = u;
  }
  static __device__ __forceinline__ float ld1(const __nv_bfloat16* p) { return __bfloat162float(*p); }
  static __device__ __forceinline__ void st1(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
};

__device__ __forceinline__ void ld8f(const float* p, float (&f)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// Sum over the TPR threads that share a row.  256-thread blocks hold 256 / TPR rows; every thread of the
// block calls this the same number of times (rows are processed in lockstep).
template <int TPR>
__device__ __forceinline__ float row_sum(float v, float (*smem)[8]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (TPR == 32) return v;
  constexpr int kWarps = TPR / 32;
  const int sub = threadIdx.x / TPR;
  const int w = (threadIdx.x % TPR) >> 5;
  __syncthreads();  // previous use of smem is over
  if ((threadIdx.x & 31) == 0) smem[sub][w] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < kWarps; ++i) t += smem[sub][i];
  return t;
}

// A thread's columns of gamma and beta: kept over the rows where they are eight (registers), else read for each.
template <bool kKeep>
struct Affine {
  float g[kKeep ? 8 : 1], b[kKeep ? 8 : 1];
  __device__ Affine(const float* gamma, const float* beta, int at) {
    if constexpr (kKeep) {
      if (gamma && at >= 0) ld8f(gamma + at, g);
      if (beta && at >= 0) ld8f(beta + at, b);
    }
  }
  __device__ void get(const float* gamma, const float* beta, int at, float (&go)[8], float (&bo)[8]) const {
    if constexpr (kKeep) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        go[i] = g[i];
        bo[i] = b[i];
      }
    } else {
      if (gamma) ld8f(gamma + at, go);
      if (beta) ld8f(beta + at, bo);
    }
  }
};

// The column statistics that ln_fold_kernel adds to are cleared by the first block of the kernel ahead of it (NULL: they are
// added to what is there): a launch and a gap of 3 us less than with a fill.
__device__ __forceinline__ void clear_stats(float* stats, int cols) {
  if (stats != nullptr && blockIdx.x == 0)
    for (int i = threadIdx.x; i < 3 * cols; i += blockDim.x) stats[i] = 0.f;
}

// Forward.  A row lives in registers: TPR threads x K vectors of 8 elements.
template <typename T, int TPR, int K>
__global__ void __launch_bounds__(256)
ln_fwd_kernel(const T* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
              T* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, long long rows,
              int cols, float eps, int pre_act) {
  __shared__ float smem[8][8];
  constexpr int kRowsPerBlock = 256 / TPR;
  constexpr bool kFast = V8<T>::kFastMath;
  const int sub = threadIdx.x / TPR;
  const int t = threadIdx.x % TPR;
  const int nvec = cols >> 3;
  const float inv_n = 1.f / static_cast<float>(cols);
  const long long row_stride = static_cast<long long>(gridDim.x) * kRowsPerBlock;
  const Affine<K == 1> par(gamma, beta, t < nvec ? t * 8 : -1);
  typename V8<T>::Raw raw[K], nxt[K];
  {
    const long long r0 = static_cast<long long>(blockIdx.x) * kRowsPerBlock + sub;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (r0 < rows && vi < nvec) raw[k] = V8<T>::ld(x + r0 * cols + vi * 8);
    }
  }
  for (long long row0 = static_cast<long long>(blockIdx.x) * kRowsPerBlock; row0 < rows; row0 += row_stride) {
    const long long row = row0 + sub;
    const bool live = row < rows;
    {  // the next row's loads are in flight while this row is reduced and written
      const long long rn = row + row_stride;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int vi = t + k * TPR;
        if (rn < rows && vi < nvec) nxt[k] = V8<T>::ld(x + rn * cols + vi * 8);
      }
    }
    float v[K][8];
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (live && vi < nvec) {
        V8<T>::unpack(raw[k], v[k]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (pre_act == FB_ACT_GELU) v[k][i] = gelu_f<kFast>(v[k][i]);
          s += v[k][i];
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[k][i] = 0.f;
      }
    }
    const float mu = row_sum<TPR>(s, smem) * inv_n;
    float q = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (live && vi < nvec) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float d = v[k][i] - mu;
          q += d * d;
        }
      }
    }
    const float var = row_sum<TPR>(q, smem) * inv_n;
    const float rs = rsqrtf(var + eps);
    if (live && t == 0) {
      if (mean_out) mean_out[row] = mu;
      if (rstd_out) rstd_out[row] = rs;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (live && vi < nvec) {
        float g[8], b[8], o[8];
        par.get(gamma, beta, vi * 8, g, b);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          o[i] = (v[k][i] - mu) * rs * (gamma ? g[i] : 1.f) + (beta ? b[i] : 0.f);
        V8<T>::st(y + row * cols + vi * 8, o);
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) raw[k] = nxt[k];
  }
}

// Forward of norm(x + r): the residual connection in front of a normalisation, fp32 x and a sub-layer's result r of
// either type.  Bound by HBM: x and r are read once and the sum (what the backward pass needs; NULL: not kept) and y
// written, where an addition of its own writes the sum and this kernel's like reads it again.
template <typename R, int TPR, int K>
__global__ void __launch_bounds__(256)
ln_add_fwd_kernel(const float* __restrict__ x, const R* __restrict__ r, const float* __restrict__ gamma,
                  const float* __restrict__ beta, float* __restrict__ sum, float* __restrict__ y,
                  float* __restrict__ mean_out, float* __restrict__ rstd_out, long long rows, int cols, float eps) {
  __shared__ float smem[8][8];
  constexpr int kRowsPerBlock = 256 / TPR;
  const int sub = threadIdx.x / TPR;
  const int t = threadIdx.x % TPR;
  const int nvec = cols >> 3;
  const float inv_n = 1.f / static_cast<float>(cols);
  const long long row_stride = static_cast<long long>(gridDim.x) * kRowsPerBlock;
  const Affine<K == 1> par(gamma, beta, t < nvec ? t * 8 : -1);
  V8<float>::Raw raw[K], nxt[K];
  typename V8<R>::Raw res[K], res_nxt[K];
  {
    const long long r0 = static_cast<long long>(blockIdx.x) * kRowsPerBlock + sub;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (r0 < rows && vi < nvec) {
        raw[k] = V8<float>::ld(x + r0 * cols + vi * 8);
        res[k] = V8<R>::ld(r + r0 * cols + vi * 8);
      }
    }
  }
  for (long long row0 = static_cast<long long>(blockIdx.x) * kRowsPerBlock; row0 < rows; row0 += row_stride) {
    const long long row = row0 + sub;
    const bool live = row < rows;
    {  // the next row's loads are in flight while this one is reduced and written
      const long long rn = row + row_stride;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int vi = t + k * TPR;
        if (rn < rows && vi < nvec) {
          nxt[k] = V8<float>::ld(x + rn * cols + vi * 8);
          res_nxt[k] = V8<R>::ld(r + rn * cols + vi * 8);
        }
      }
    }
    float v[K][8];
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (live && vi < nvec) {
        float w[8];
        V8<float>::unpack(raw[k], v[k]);
        V8<R>::unpack(res[k], w);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          v[k][i] += w[i];
          s += v[k][i];
        }
        if (sum != nullptr) V8<float>::st(sum + row * cols + vi * 8, v[k]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[k][i] = 0.f;
      }
    }
    const float mu = row_sum<TPR>(s, smem) * inv_n;
    float q = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (live && vi < nvec) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float d = v[k][i] - mu;
          q += d * d;
        }
      }
    }
    const float var = row_sum<TPR>(q, smem) * inv_n;
    const float rs = rsqrtf(var + eps);
    if (live && t == 0) {
      mean_out[row] = mu;
      rstd_out[row] = rs;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (live && vi < nvec) {
        float g[8], b[8], o[8];
        par.get(gamma, beta, vi * 8, g, b);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          o[i] = (v[k][i] - mu) * rs * (gamma ? g[i] : 1.f) + (beta ? b[i] : 0.f);
        V8<float>::st(y + row * cols + vi * 8, o);
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      raw[k] = nxt[k];
      res[k] = res_nxt[k];
    }
  }
}

__device__ __forceinline__ void ld_pairs_f32(const float* p, float2 (&o)[4]);

// Forward, one WARP per row (bf16, 1024..4096 columns): a lane keeps its K 16-byte vectors packed in registers,
// all K loads are issued back to back (up to 8 KB in flight per warp), the statistics are one pass of shifted sums
// (x - c with c = the row's first element) reduced by warp shuffles, and there is no block barrier at all: warps
// stream rows independently.  Packed fp32x2 arithmetic.  gamma and beta lie in shared memory, quads of columns side by
// side (the even ones of a parameter, then the odd ones), so that a warp's 16-byte reads are free of bank conflicts: read
// through L1 for each row, beside the rows that stream past, they were a third of the time.  8192 x 4096 36.1 -> 24.9 us (a copy
// of the rows takes 22).
// W > 1, few rows: a block per row.  Latency is all there is then, so W warps find the same statistics (the same sums in
// the same order: the same bits) and each writes the vectors k % W of its number, whose gamma and beta it asks for
// beforehand.
template <int K, int W = 1>
__global__ void __launch_bounds__(256, 2)
ln_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                   __nv_bfloat16* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out,
                   long long rows, int cols, float eps) {
  if constexpr (W > 1) {
    ptx::grid_launch_dependents();
    ptx::grid_wait();
  }
  const int lane = threadIdx.x & 31;
  const int nvec = cols >> 3;
  const float inv_n = 1.f / static_cast<float>(cols);
  const int part = W > 1 ? threadIdx.x >> 5 : 0;
  const long long warp_id = W > 1 ? blockIdx.x : (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = W > 1 ? gridDim.x : (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  constexpr int kOwn = W > 1 ? K / W : 1;
  float2 own_g[kOwn][4], own_b[kOwn][4];
  extern __shared__ float4 affine[];  // W == 1: gamma's even quads, odd quads, beta's even quads, odd quads
  if constexpr (W == 1) {
    for (int i = threadIdx.x; i < 2 * nvec; i += 256) {
      const int at = (i & 1) * nvec + (i >> 1);
      affine[at] = gamma ? *reinterpret_cast<const float4*>(gamma + 4 * i) : make_float4(1.f, 1.f, 1.f, 1.f);
      affine[2 * nvec + at] = beta ? *reinterpret_cast<const float4*>(beta + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
  }
  for (long long row = warp_id; row < rows; row += nwarps) {
    const __nv_bfloat16* xr = x + row * cols;
    uint4 raw[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = lane + 32 * k;
      raw[k] = vi < nvec ? *reinterpret_cast<const uint4*>(xr + vi * 8) : make_uint4(0u, 0u, 0u, 0u);
    }
    if constexpr (W > 1) {
#pragma unroll
      for (int i = 0; i < kOwn; ++i) {
        const int vi = lane + 32 * (part + W * i);
        if (gamma && vi < nvec) ld_pairs_f32(gamma + vi * 8, own_g[i]);
        if (beta && vi < nvec) ld_pairs_f32(beta + vi * 8, own_b[i]);
      }
    }
    // c = element 0 of the row = low half of lane 0's first word
    const float c = __uint_as_float(__shfl_sync(0xffffffffu, raw[0].x, 0) << 16);
    const float2 nc = make_float2(-c, -c);
    float2 s2 = make_float2(0.f, 0.f), q2 = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (lane + 32 * k < nvec) {
        const uint32_t w[4] = {raw[k].x, raw[k].y, raw[k].z, raw[k].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 v = make_float2(__uint_as_float(w[e] << 16), __uint_as_float(w[e] & 0xffff0000u));
          const float2 d = __fadd2_rn(v, nc);
          s2 = __fadd2_rn(s2, d);
          q2 = __ffma2_rn(d, d, q2);
        }
      }
    }
    float s = s2.x + s2.y, q = q2.x + q2.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      q += __shfl_xor_sync(0xffffffffu, q, o);
    }
    const float ms = s * inv_n;
    const float var = fmaxf(q * inv_n - ms * ms, 0.f);
    const float mu = c + ms;
    const float rs = rsqrtf(var + eps);
    if (lane == 0 && part == 0) {
      if (mean_out) mean_out[row] = mu;
      if (rstd_out) rstd_out[row] = rs;
    }
    const float2 rs2 = make_float2(rs, rs), sh2 = make_float2(-mu * rs, -mu * rs);
    __nv_bfloat16* yr = y + row * cols;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = lane + 32 * k;
      if (vi < nvec && (W == 1 || k % W == part)) {
        const uint32_t w[4] = {raw[k].x, raw[k].y, raw[k].z, raw[k].w};
        float2 g[4], b[4];
        if constexpr (W > 1) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            g[e] = gamma ? own_g[k / W][e] : make_float2(1.f, 1.f);
            b[e] = beta ? own_b[k / W][e] : make_float2(0.f, 0.f);
          }
        } else {
          const float4 g0 = affine[vi], g1 = affine[nvec + vi], b0 = affine[2 * nvec + vi], b1 = affine[3 * nvec + vi];
          g[0] = make_float2(g0.x, g0.y); g[1] = make_float2(g0.z, g0.w);
          g[2] = make_float2(g1.x, g1.y); g[3] = make_float2(g1.z, g1.w);
          b[0] = make_float2(b0.x, b0.y); b[1] = make_float2(b0.z, b0.w);
          b[2] = make_float2(b1.x, b1.y); b[3] = make_float2(b1.z, b1.w);
        }
        uint4 out;
        uint32_t* ow = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 v = make_float2(__uint_as_float(w[e] << 16), __uint_as_float(w[e] & 0xffff0000u));
          const float2 o = __ffma2_rn(__ffma2_rn(v, rs2, sh2), g[e], b[e]);
          const __nv_bfloat162 pk = __float22bfloat162_rn(o);
          ow[e] = *reinterpret_cast<const uint32_t*>(&pk);
        }
        *reinterpret_cast<uint4*>(yr + vi * 8) = out;
      }
    }
  }
}

template <int N>
__device__ __forceinline__ void st_piece(float* p, const float* v) {
  if constexpr (N == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  else *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

// Backward.  x and dy stay packed in registers between the statistics pass and the output pass; the
// three column partials (dy*xhat, dy, dx) accumulate in registers over all rows the block visits and are
// written once to partial[blockIdx][3][cols].  kLow: dx once more in bf16, the gradient of a residual's branch (K = 4: if there
// is a dx_low; that instance spills least).
// Bound by loads in flight, hence three blocks per SM where a thread holds one vector, and for few rows by the rows of a
// block adding up, which they do in shared memory (one after the other through global memory each waited for the one
// before).  fp32: 128 x 256 10.9 -> 4.4 us, 1024 x 1024 13.1 -> 8.8, 8192 x 1024 with dx_low 36.8 -> 31.7.
template <typename T, int TPR, int K, bool kLow>
__global__ void __launch_bounds__(256, K == 1 ? 3 : 2)
ln_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ act_grad,
              const float* __restrict__ gamma, const float* __restrict__ mean, const float* __restrict__ rstd,
              T* __restrict__ dx, __nv_bfloat16* __restrict__ dx_low, float* __restrict__ partial, long long rows,
              int cols, int pre_act, int want_colsum, float* __restrict__ clear) {
  clear_stats(clear, cols);
  __shared__ float smem[8][8];
  constexpr int kRowsPerBlock = 256 / TPR;
  constexpr bool kFast = V8<T>::kFastMath;
  const int sub = threadIdx.x / TPR;
  const int t = threadIdx.x % TPR;
  const int nvec = cols >> 3;
  const float inv_n = 1.f / static_cast<float>(cols);
  float acc_g[K][8], acc_b[K][8], acc_c[K][8];
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc_g[k][i] = acc_b[k][i] = acc_c[k][i] = 0.f;

  const long long row_stride = static_cast<long long>(gridDim.x) * kRowsPerBlock;
  typename V8<T>::Raw xr[K], gr[K], xn[K], gn[K];
  {
    const long long r0 = static_cast<long long>(blockIdx.x) * kRowsPerBlock + sub;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (r0 < rows && vi < nvec) {
        xr[k] = V8<T>::ld(x + r0 * cols + vi * 8);
        gr[k] = V8<T>::ld(dy + r0 * cols + vi * 8);
      }
    }
  }
  for (long long row0 = static_cast<long long>(blockIdx.x) * kRowsPerBlock; row0 < rows; row0 += row_stride) {
    const long long row = row0 + sub;
    const bool live = row < rows;
    {  // prefetch the next row while this one is processed
      const long long rn = row + row_stride;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int vi = t + k * TPR;
        if (rn < rows && vi < nvec) {
          xn[k] = V8<T>::ld(x + rn * cols + vi * 8);
          gn[k] = V8<T>::ld(dy + rn * cols + vi * 8);
        }
      }
    }
    const float mu = live ? mean[row] : 0.f;
    const float rs = live ? rstd[row] : 0.f;
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (live && vi < nvec) {
        float xv[8], gv[8], w[8];
        V8<T>::unpack(xr[k], xv);
        V8<T>::unpack(gr[k], gv);
        if (gamma) ld8f(gamma + vi * 8, w);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float a = pre_act == FB_ACT_GELU ? gelu_f<kFast>(xv[i]) : xv[i];
          const float h = (a - mu) * rs;
          const float d = gv[i] * (gamma ? w[i] : 1.f);
          acc_g[k][i] += gv[i] * h;
          acc_b[k][i] += gv[i];
          s1 += d;
          s2 += d * h;
        }
      }
    }
    const float m1 = row_sum<TPR>(s1, smem) * inv_n;
    const float m2 = row_sum<TPR>(s2, smem) * inv_n;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (live && vi < nvec) {
        float xv[8], gv[8], w[8], o[8];
        V8<T>::unpack(xr[k], xv);
        V8<T>::unpack(gr[k], gv);
        if (gamma) ld8f(gamma + vi * 8, w);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float a = xv[i], da = 1.f;
          if (pre_act == FB_ACT_GELU) gelu_both<kFast>(xv[i], a, da);
          const float h = (a - mu) * rs;
          const float d = gv[i] * (gamma ? w[i] : 1.f);
          o[i] = rs * (d - m1 - h * m2) * da;
        }
        if (act_grad != nullptr) {  // x holds act(z); its derivative was stored by the producer
          float ag[8];
          V8<T>::unpack(V8<T>::ld(act_grad + row * cols + vi * 8), ag);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] *= ag[i];
        }
        if (want_colsum) {
#pragma unroll
          for (int i = 0; i < 8; ++i) acc_c[k][i] += o[i];
        }
        V8<T>::st(dx + row * cols + vi * 8, o);
        if (kLow && (K < 4 || dx_low != nullptr)) V8<__nv_bfloat16>::st(dx_low + row * cols + vi * 8, o);
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      xr[k] = xn[k];
      gr[k] = gn[k];
    }
  }

  // ---- column partials of this block: partial[blockIdx][3][cols]
  float* pg = partial + static_cast<long long>(blockIdx.x) * 3 * cols;
  float* pb = pg + cols;
  float* pc = pb + cols;
  if constexpr (kRowsPerBlock == 1) {
    // K = 2 in pairs: 16-byte pieces cost the loop above 56 bytes of spills (fp32, 8192 x 3072 106 us instead of 99, though
    // 300 x 4096 20.6 instead of 22.0); K = 4 spills either way (8192 x 8192 386 us, in pairs 431, element by element 520)
    constexpr int kPiece = K == 2 ? 2 : 4;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = t + k * TPR;
      if (vi >= nvec) continue;
#pragma unroll
      for (int i = 0; i < 8; i += kPiece) {
        st_piece<kPiece>(pg + vi * 8 + i, &acc_g[k][i]);
        st_piece<kPiece>(pb + vi * 8 + i, &acc_b[k][i]);
        st_piece<kPiece>(pc + vi * 8 + i, &acc_c[k][i]);
      }
    }
  } else {
    // Several row slots own the same columns: they add up in shared memory, one slot at a time, and the last one stores.
    __shared__ float cols_sum[3][K * TPR * 8];
#pragma unroll 1
    for (int slot = 0; slot < kRowsPerBlock; ++slot) {
      __syncthreads();
      if (sub != slot) continue;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int vi = t + k * TPR;
        if (vi >= nvec) continue;
        if (slot > 0) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int at = (k * 8 + i) * TPR + t;
            acc_g[k][i] = cols_sum[0][at] + acc_g[k][i];
            acc_b[k][i] = cols_sum[1][at] + acc_b[k][i];
            acc_c[k][i] = cols_sum[2][at] + acc_c[k][i];
          }
        }
        if (slot + 1 == kRowsPerBlock) {
          V8<float>::st(pg + vi * 8, acc_g[k]);
          V8<float>::st(pb + vi * 8, acc_b[k]);
          V8<float>::st(pc + vi * 8, acc_c[k]);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int at = (k * 8 + i) * TPR + t;
            cols_sum[0][at] = acc_g[k][i];
            cols_sum[1][at] = acc_b[k][i];
            cols_sum[2][at] = acc_c[k][i];
          }
        }
      }
    }
  }
}

// ----------------------------------------------------------------------------------------------------
// Wide rows (2 KB .. 8 KB of bf16 / 16 KB of fp32, i.e. up to 4096 columns): shared-memory ring fed by bulk
// async copies, organised for few instructions per element.
//
// Measured on the register-tiled kernels above and on a first ring version: with ~30-40 instructions per
// element these kernels are bound by instruction issue (issue slots 55-60 % busy, the rest barrier / dependency
// stalls), not by HBM.  So:
//   * a thread owns 16 elements of a row (two 16-byte vectors of bf16), which halves the per-row fixed cost
//     (shuffles, shared-memory exchange, barrier) per element;
//   * the forward needs ONE reduction per row: sums of (x - c) and (x - c)^2 with c = the row's first element
//     (shifted sums: no cancellation unless the row's spread is tiny against |x0 - mean|);
//   * a 512-thread block is two independent groups of 256 threads, each with its own ring, mbarriers and named
//     barrier, so one group's barrier wait overlaps the other group's arithmetic;
//   * rows arrive by cp.async.bulk into the ring, up to three rows ahead per group: no registers or scoreboards
//     are tied up by prefetched data;
//   * the arithmetic is packed fp32x2 (FFMA2 / FADD2 / FMUL2).
// Measured at 8192 x 4096 bf16: backward 64-66 us against 128 us for the register-tiled kernel; the forward
// (42-45 us) does not beat the register-tiled forward (39-40 us), so the forward ring is opt-in
// (FERRUM_LN_RING_FWD=1) and the default forward stays on the register-tiled kernel.  A slot is refilled at the top of the iteration after the one that read it (every
//     thread of the group has passed that iteration's barrier by then).
// Packed fp32x2 arithmetic (Blackwell FFMA2 / FADD2 / FMUL2): one issue slot does two fp32 operations, which
// matters here because these kernels are bound by instruction issue, not by HBM.
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 f2s(float a) { return make_float2(a, a); }
template <typename T>
__device__ __forceinline__ void unpack_pairs(const typename V8<T>::Raw& r, float2 (&p)[4]) {
  float f[8];
  V8<T>::unpack(r, f);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = make_float2(f[2 * i], f[2 * i + 1]);
}
template <typename T>
__device__ __forceinline__ void store_pairs(T* dst, const float2 (&p)[4]) {
  float f[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = p[i].x;
    f[2 * i + 1] = p[i].y;
  }
  V8<T>::st(dst, f);
}
__device__ __forceinline__ void ld_pairs_f32(const float* p, float2 (&o)[4]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  o[0] = make_float2(a.x, a.y);
  o[1] = make_float2(a.z, a.w);
  o[2] = make_float2(b.x, b.y);
  o[3] = make_float2(b.z, b.w);
}
// Sum of (a, b) over the eight warps of a 256-thread group: lane 0 of every warp has written its partial to
// slot[warp]; after the group barrier every thread folds the eight partials with three shuffles.
__device__ __forceinline__ float2 fold8(const float2* slot, int lane) {
  float2 v = slot[lane & 7];
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

constexpr int kRingThreads = 512;
constexpr int kGroupThreads = 256;
constexpr int kMaxRingStages = 4;  // per group (measured: 2 .. 6 stages perform alike; the kernels are issue-bound)
constexpr int kStatRows = 128;   // per-group cache of mean / rstd (backward)

struct RingCtl {
  uint64_t full[2][kMaxRingStages];
  int abort_flag;
};

__device__ __forceinline__ void group_sync(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(kGroupThreads) : "memory");
}
__device__ __forceinline__ bool ring_wait(RingCtl* ctl, int group, int i, int stages) {
  return ptx::mbar_wait(&ctl->full[group][i % stages], static_cast<uint32_t>((i / stages) & 1), &ctl->abort_flag,
                        2000000000ull);
}
// Before a group with copies in flight may exit, let them land (bounded).
__device__ __forceinline__ void ring_drain(RingCtl* ctl, int group, int issued, int consumed, int stages) {
  for (int i = consumed; i < issued; ++i) {
    const uint64_t t0 = ptx::globaltimer();
    while (!ptx::mbar_try_wait(&ctl->full[group][i % stages], static_cast<uint32_t>((i / stages) & 1))) {
      if (ptx::globaltimer() - t0 > 2000000000ull) break;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kRingThreads, sizeof(T) == 2 ? 2 : 1)
ln_fwd_ring_kernel(const T* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                   T* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, long long rows,
                   int cols, float eps, int pre_act, int stages, int32_t* status) {
  extern __shared__ __align__(128) uint8_t ring[];
  __shared__ RingCtl ctl;
  __shared__ float2 red[2][2][8];
  constexpr bool kFast = V8<T>::kFastMath;
  const int group = threadIdx.x >> 8, t = threadIdx.x & 255, lane = t & 31, warp = t >> 5;
  const int nvec = cols >> 3;
  const uint32_t row_bytes = static_cast<uint32_t>(cols) * sizeof(T);
  uint8_t* my_ring = ring + group * stages * row_bytes;
  const float inv_n = 1.f / static_cast<float>(cols);
  // the block's rows are first + j * stride; group g takes j = 2 i + g
  const long long first = blockIdx.x, stride = gridDim.x;
  const long long n_block = first < rows ? (rows - first + stride - 1) / stride : 0;
  const int n_mine = static_cast<int>((n_block - group + 1) / 2);
  auto row_of = [&](int i) { return first + (2LL * i + group) * stride; };
  if (threadIdx.x == 0) {
    ctl.abort_flag = 0;
    for (int g = 0; g < 2; ++g)
      for (int s = 0; s < stages; ++s) ptx::mbar_init(&ctl.full[g][s], 1);
    ptx::fence_mbar_init();
  }
  __syncthreads();
  auto issue = [&](int idx) {
    const int sl = idx % stages;
    ptx::mbar_arrive_expect_tx(&ctl.full[group][sl], row_bytes);
    ptx::bulk_load_1d(my_ring + sl * row_bytes, x + row_of(idx) * cols, row_bytes, &ctl.full[group][sl]);
  };
  int issued = 0;
  if (t == 0)
    for (; issued < stages - 1 && issued < n_mine; ++issued) issue(issued);

  const bool has[2] = {t < nvec, t + kGroupThreads < nvec};
  int i = 0, par = 0;
  for (; i < n_mine; ++i) {
    const long long row = row_of(i);
    if (t == 0 && issued < n_mine) issue(issued++);  // refills the slot that iteration i - 1 read
    if (!ring_wait(&ctl, group, i, stages)) break;
    const T* src = reinterpret_cast<const T*>(my_ring + (i % stages) * row_bytes);
    float2 v[2][4];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (has[k]) {
        unpack_pairs<T>(V8<T>::ld(src + (t + k * kGroupThreads) * 8), v[k]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[k][e] = f2s(0.f);
      }
    }
    float c = V8<T>::ld1(src);
    if (pre_act == FB_ACT_GELU) {
      c = gelu_f<kFast>(c);
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int e = 0; e < 4; ++e) v[k][e] = f2(gelu_f<kFast>(v[k][e].x), gelu_f<kFast>(v[k][e].y));
    }
    const float2 nc = f2s(-c);
    float2 s2 = f2s(0.f), q2 = f2s(0.f);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (has[k]) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 d = __fadd2_rn(v[k][e], nc);
          s2 = __fadd2_rn(s2, d);
          q2 = __ffma2_rn(d, d, q2);
        }
      }
    }
    float s = s2.x + s2.y, q = q2.x + q2.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      q += __shfl_xor_sync(0xffffffffu, q, o);
    }
    if (lane == 0) red[group][par][warp] = make_float2(s, q);
    group_sync(group);
    const float2 tot = fold8(red[group][par], lane);
    par ^= 1;
    const float ms = tot.x * inv_n;                       // mean of (x - c)
    const float var = fmaxf(tot.y * inv_n - ms * ms, 0.f);
    const float mu = c + ms;
    const float rs = rsqrtf(var + eps);
    if (t == 0) {
      if (mean_out) mean_out[row] = mu;
      if (rstd_out) rstd_out[row] = rs;
    }
    const float2 rs2 = f2s(rs), shift2 = f2s(-mu * rs);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int vi = t + k * kGroupThreads;
      if (has[k]) {
        float2 g[4], b[4], o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          g[e] = f2s(1.f);
          b[e] = f2s(0.f);
        }
        if (gamma) ld_pairs_f32(gamma + vi * 8, g);
        if (beta) ld_pairs_f32(beta + vi * 8, b);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = __ffma2_rn(__ffma2_rn(v[k][e], rs2, shift2), g[e], b[e]);
        store_pairs<T>(y + row * cols + vi * 8, o);
      }
    }
  }
  if (i < n_mine && t == 0) {  // a wait gave up
    report_status(status, kStatusGemmTimeout, 31, blockIdx.x, i);
    ring_drain(&ctl, group, issued, i, stages);
  }
}

// Backward with the activation derivative (if any) given as a tensor: bf16, up to 4096 columns.  A slot
// holds the dy, x and act_grad rows; gamma and the three column accumulators stay in registers; mean / rstd
// of a group's rows are cached in shared memory up front; a row costs one group barrier.  Column partials:
// one row of partial[] per GROUP (2 * gridDim.x rows in all).
__global__ void __launch_bounds__(kRingThreads, 1)
ln_bwd_ring_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const __nv_bfloat16* __restrict__ act_grad, const float* __restrict__ gamma,
                   const float* __restrict__ mean, const float* __restrict__ rstd, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ partial, long long rows, int cols, int want_colsum, int stages,
                   int32_t* status, float* __restrict__ clear) {
  clear_stats(clear, cols);
  using V = V8<__nv_bfloat16>;
  extern __shared__ __align__(128) uint8_t ring[];
  __shared__ RingCtl ctl;
  __shared__ float2 red[2][2][8];
  __shared__ float2 stat[2][kStatRows];
  const int group = threadIdx.x >> 8, t = threadIdx.x & 255, lane = t & 31, warp = t >> 5;
  const int nvec = cols >> 3;
  const bool use_ag = act_grad != nullptr;
  const uint32_t row_bytes = static_cast<uint32_t>(cols) * 2u;
  const uint32_t slot_bytes = row_bytes * (use_ag ? 3u : 2u);
  uint8_t* my_ring = ring + group * stages * slot_bytes;
  const float inv_n = 1.f / static_cast<float>(cols);
  const long long first = blockIdx.x, stride = gridDim.x;
  const long long n_block = first < rows ? (rows - first + stride - 1) / stride : 0;
  const int n_mine = static_cast<int>((n_block - group + 1) / 2);
  auto row_of = [&](int i) { return first + (2LL * i + group) * stride; };

  if (threadIdx.x == 0) {
    ctl.abort_flag = 0;
    for (int g = 0; g < 2; ++g)
      for (int s = 0; s < stages; ++s) ptx::mbar_init(&ctl.full[g][s], 1);
    ptx::fence_mbar_init();
  }
  for (int r = t; r < n_mine && r < kStatRows; r += kGroupThreads)
    stat[group][r] = make_float2(mean[row_of(r)], rstd[row_of(r)]);
  __syncthreads();
  auto issue = [&](int idx) {
    const int sl = idx % stages;
    uint8_t* dst = my_ring + sl * slot_bytes;
    const long long off = row_of(idx) * cols;
    ptx::mbar_arrive_expect_tx(&ctl.full[group][sl], slot_bytes);
    ptx::bulk_load_1d(dst, dy + off, row_bytes, &ctl.full[group][sl]);
    ptx::bulk_load_1d(dst + row_bytes, x + off, row_bytes, &ctl.full[group][sl]);
    if (use_ag) ptx::bulk_load_1d(dst + 2 * row_bytes, act_grad + off, row_bytes, &ctl.full[group][sl]);
  };
  int issued = 0;
  if (t == 0)
    for (; issued < stages - 1 && issued < n_mine; ++issued) issue(issued);

  const bool has[2] = {t < nvec, t + kGroupThreads < nvec};
  float2 w[2][4], acc_g[2][4], acc_b[2][4], acc_c[2][4];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      w[k][e] = f2s(1.f);
      acc_g[k][e] = acc_b[k][e] = acc_c[k][e] = f2s(0.f);
    }
    if (has[k] && gamma != nullptr) ld_pairs_f32(gamma + (t + k * kGroupThreads) * 8, w[k]);
  }

  int i = 0, par = 0;
  for (; i < n_mine; ++i) {
    const long long row = row_of(i);
    if (t == 0 && issued < n_mine) issue(issued++);  // refills the slot that iteration i - 1 read
    if (!ring_wait(&ctl, group, i, stages)) break;
    const float2 st = i < kStatRows ? stat[group][i] : make_float2(mean[row], rstd[row]);
    const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(my_ring + (i % stages) * slot_bytes);
    float2 d[2][4], h[2][4];
    const float2 rs2 = f2s(st.y), shift2 = f2s(-st.x * st.y);
    float2 s1 = f2s(0.f), s2 = f2s(0.f);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (has[k]) {
        const int vi = t + k * kGroupThreads;
        unpack_pairs<__nv_bfloat16>(V::ld(src + vi * 8), d[k]);
        unpack_pairs<__nv_bfloat16>(V::ld(src + cols + vi * 8), h[k]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          h[k][e] = __ffma2_rn(h[k][e], rs2, shift2);
          acc_b[k][e] = __fadd2_rn(acc_b[k][e], d[k][e]);
          acc_g[k][e] = __ffma2_rn(d[k][e], h[k][e], acc_g[k][e]);
          d[k][e] = __fmul2_rn(d[k][e], w[k][e]);  // d = dy * gamma
          s1 = __fadd2_rn(s1, d[k][e]);
          s2 = __ffma2_rn(d[k][e], h[k][e], s2);
        }
      }
    }
    float a1 = s1.x + s1.y, a2 = s2.x + s2.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a1 += __shfl_xor_sync(0xffffffffu, a1, o);
      a2 += __shfl_xor_sync(0xffffffffu, a2, o);
    }
    if (lane == 0) red[group][par][warp] = make_float2(a1, a2);
    group_sync(group);
    const float2 tot = fold8(red[group][par], lane);
    par ^= 1;
    // o = rstd * (d - m1 - h m2) with rstd folded into the two means
    const float2 nm1 = f2s(-tot.x * inv_n * st.y), nm2 = f2s(-tot.y * inv_n * st.y);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (has[k]) {
        const int vi = t + k * kGroupThreads;
        float2 o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = __ffma2_rn(h[k][e], nm2, __ffma2_rn(d[k][e], rs2, nm1));
        if (use_ag) {
          float2 ag[4];
          unpack_pairs<__nv_bfloat16>(V::ld(src + 2 * cols + vi * 8), ag);
#pragma unroll
          for (int e = 0; e < 4; ++e) o[e] = __fmul2_rn(o[e], ag[e]);
        }
        if (want_colsum) {
#pragma unroll
          for (int e = 0; e < 4; ++e) acc_c[k][e] = __fadd2_rn(acc_c[k][e], o[e]);
        }
        store_pairs<__nv_bfloat16>(dx + row * cols + vi * 8, o);
      }
    }
  }
  if (i < n_mine && t == 0) {
    report_status(status, kStatusGemmTimeout, 32, blockIdx.x, i);
    ring_drain(&ctl, group, issued, i, stages);
  }
  float* base = partial + (2LL * blockIdx.x + group) * 3 * cols;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (has[k]) {
      float* pg = base + (t + k * kGroupThreads) * 8;
      float* pb = pg + cols;
      float* pc = pb + cols;
      *reinterpret_cast<float4*>(pg) = make_float4(acc_g[k][0].x, acc_g[k][0].y, acc_g[k][1].x, acc_g[k][1].y);
      *reinterpret_cast<float4*>(pg + 4) = make_float4(acc_g[k][2].x, acc_g[k][2].y, acc_g[k][3].x, acc_g[k][3].y);
      *reinterpret_cast<float4*>(pb) = make_float4(acc_b[k][0].x, acc_b[k][0].y, acc_b[k][1].x, acc_b[k][1].y);
      *reinterpret_cast<float4*>(pb + 4) = make_float4(acc_b[k][2].x, acc_b[k][2].y, acc_b[k][3].x, acc_b[k][3].y);
      *reinterpret_cast<float4*>(pc) = make_float4(acc_c[k][0].x, acc_c[k][0].y, acc_c[k][1].x, acc_c[k][1].y);
      *reinterpret_cast<float4*>(pc + 4) = make_float4(acc_c[k][2].x, acc_c[k][2].y, acc_c[k][3].x, acc_c[k][3].y);
    }
  }
}

// Fold partial[nblk][3*cols] into stats[3*cols] (accumulated into): block = 128 columns x a chunk of the
// nblk rows, lanes own 4 adjacent columns, partials leave with one atomicAdd per column per block.  (Without
// atomics, a cluster or a block to a column range, it took 4.5 to 5.5 us for 1024 columns instead of 2.9: too few blocks.)  kVec: 16-byte loads
// (ncols a multiple of 4, partial on a 16-byte address).
template <bool kVec>
__global__ void __launch_bounds__(256)
ln_fold_kernel(const float* __restrict__ partial, float* __restrict__ stats, int nblk, int ncols,
               int rows_per_block) {
  __shared__ float sm[8][128];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = blockIdx.x * 128 + lane * 4;
  const int r_lo = blockIdx.y * rows_per_block;
  const int r_hi = min(nblk, r_lo + rows_per_block);
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (!kVec) {
    for (int r = r_lo + warp; r < r_hi; r += 8) {
      const float* v = partial + static_cast<long long>(r) * ncols + c0;
      if (c0 < ncols) a.x += v[0];
      if (c0 + 1 < ncols) a.y += v[1];
      if (c0 + 2 < ncols) a.z += v[2];
      if (c0 + 3 < ncols) a.w += v[3];
    }
  } else if (c0 < ncols) {
    for (int r = r_lo + warp; r < r_hi; r += 8) {
      const float4 v = *reinterpret_cast<const float4*>(partial + static_cast<long long>(r) * ncols + c0);
      a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    }
  }
  sm[warp][lane * 4 + 0] = a.x;
  sm[warp][lane * 4 + 1] = a.y;
  sm[warp][lane * 4 + 2] = a.z;
  sm[warp][lane * 4 + 3] = a.w;
  __syncthreads();
  if (threadIdx.x < 128) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += sm[w][threadIdx.x];
    const int c = blockIdx.x * 128 + threadIdx.x;
    if (c < ncols) atomicAdd(stats + c, s);
  }
}

// ---------------------------------------------------------------- rows of any width and alignment in registers
// Widths that are no multiple of 8 (or bases off 16 bytes): TPR threads share a row, thread t owns columns t, t + TPR,
// ...  (K of them, in registers), so every access of a warp is one contiguous run whatever the row's address.  A row is
// read once; the column sums stay in registers over a block's rows, meet in shared memory and then in ln_fold_kernel.
// Bound by latency at few rows and by the 2-byte accesses at many.  777 x 1001 bf16, against three passes over the row and
// an atomic per element and column sum: forward 6.6 -> 5.6 us, backward 18.7 -> 9.2 + 2.8 (fold).
template <typename T, int TPR, int K>
__global__ void __launch_bounds__(256)
ln_fwd_any_kernel(const T* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                  T* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, long long rows, int cols,
                  float eps, int pre_act) {
  __shared__ float smem[8][8];
  constexpr int kRows = 256 / TPR;
  const int sub = threadIdx.x / TPR, t = threadIdx.x % TPR;
  for (long long row0 = static_cast<long long>(blockIdx.x) * kRows; row0 < rows;
       row0 += static_cast<long long>(gridDim.x) * kRows) {
    const long long row = row0 + sub;
    const bool live = row < rows;
    const T* xr = x + (live ? row : 0) * cols;
    float v[K], s = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int c = t + k * TPR;
      v[k] = live && c < cols ? V8<T>::ld1(xr + c) : 0.f;
    }
    if (pre_act == FB_ACT_GELU) {
#pragma unroll
      for (int k = 0; k < K; ++k) v[k] = gelu_f<false>(v[k]);  // of a padding zero: zero
    }
#pragma unroll
    for (int k = 0; k < K; ++k) s += v[k];
    const float mu = row_sum<TPR>(s, smem) / cols;
    float q = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (t + k * TPR < cols) q += (v[k] - mu) * (v[k] - mu);
    const float rs = rsqrtf(row_sum<TPR>(q, smem) / cols + eps);
    if (live && t == 0) {
      if (mean_out) mean_out[row] = mu;
      if (rstd_out) rstd_out[row] = rs;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int c = t + k * TPR;
      if (live && c < cols)
        V8<T>::st1(y + row * cols + c, (v[k] - mu) * rs * (gamma ? gamma[c] : 1.f) + (beta ? beta[c] : 0.f));
    }
  }
}

// partial[blockIdx][3][cols]: d_gamma, d_beta and the column sum of dx over the block's rows.
template <typename T, int TPR, int K>
__global__ void __launch_bounds__(256)
ln_bwd_any_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ act_grad,
                  const float* __restrict__ gamma, const float* __restrict__ mean, const float* __restrict__ rstd,
                  T* __restrict__ dx, float* __restrict__ partial, long long rows, int cols, int pre_act,
                  int want_colsum, float* __restrict__ clear) {
  clear_stats(clear, cols);
  __shared__ float smem[8][8];
  constexpr int kRows = 256 / TPR;
  const int sub = threadIdx.x / TPR, t = threadIdx.x % TPR;
  float acc_g[K], acc_b[K], acc_c[K];
#pragma unroll
  for (int k = 0; k < K; ++k) acc_g[k] = acc_b[k] = acc_c[k] = 0.f;
  for (long long row0 = static_cast<long long>(blockIdx.x) * kRows; row0 < rows;
       row0 += static_cast<long long>(gridDim.x) * kRows) {
    const long long row = row0 + sub;
    const bool live = row < rows;
    const long long at = (live ? row : 0) * cols;
    const float mu = live ? mean[row] : 0.f, rs = live ? rstd[row] : 0.f;
    float h[K], d[K], da[K], s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int c = t + k * TPR;
      const bool in = live && c < cols;
      h[k] = in ? V8<T>::ld1(x + at + c) : 0.f;
      d[k] = in ? V8<T>::ld1(dy + at + c) : 0.f;
      da[k] = act_grad != nullptr && in ? V8<T>::ld1(act_grad + at + c) : 1.f;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int c = t + k * TPR;
      if (pre_act == FB_ACT_GELU) gelu_both<false>(h[k], h[k], da[k]);
      h[k] = live && c < cols ? (h[k] - mu) * rs : 0.f;
      acc_g[k] += d[k] * h[k];
      acc_b[k] += d[k];
      if (gamma != nullptr && c < cols) d[k] *= gamma[c];
      s1 += d[k];
      s2 += d[k] * h[k];
    }
    const float m1 = row_sum<TPR>(s1, smem) / cols, m2 = row_sum<TPR>(s2, smem) / cols;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int c = t + k * TPR;
      if (!live || c >= cols) continue;
      const float o = rs * (d[k] - m1 - h[k] * m2) * da[k];
      acc_c[k] += o;
      V8<T>::st1(dx + at + c, o);
    }
  }
  // the thread groups of a block own the same columns: one after the other adds what the ones before left
  __shared__ float others[kRows == 1 ? 1 : 3 * K * TPR];
  float* p = partial + static_cast<long long>(blockIdx.x) * 3 * cols;
#pragma unroll
  for (int s = 0; s < kRows; ++s) {
    if (sub == s) {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        float v[3] = {acc_g[k], acc_b[k], want_colsum ? acc_c[k] : 0.f};
        const int c = t + k * TPR;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          if (s > 0) v[j] += others[(j * K + k) * TPR + t];
          if (s < kRows - 1) others[(j * K + k) * TPR + t] = v[j];
          else if (c < cols) p[j * cols + c] = v[j];
        }
      }
    }
    if (s < kRows - 1) __syncthreads();
  }
}

// ---------------------------------------------------------------- rows of any width, re-read
template <typename T>
__global__ void ln_fwd_generic(const T* __restrict__ x, const float* __restrict__ gamma,
                               const float* __restrict__ beta, T* __restrict__ y, float* __restrict__ mean_out,
                               float* __restrict__ rstd_out, long long rows, int cols, float eps, int pre_act) {
  __shared__ float smem[8][8];
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const T* xr = x + row * cols;
    float s = 0.f;
    for (int c = threadIdx.x; c < cols; c += 256) {
      float a = V8<T>::ld1(xr + c);
      if (pre_act == FB_ACT_GELU) a = gelu_f<false>(a);
      s += a;
    }
    const float mu = row_sum<256>(s, smem) / cols;
    float q = 0.f;
    for (int c = threadIdx.x; c < cols; c += 256) {
      float a = V8<T>::ld1(xr + c);
      if (pre_act == FB_ACT_GELU) a = gelu_f<false>(a);
      q += (a - mu) * (a - mu);
    }
    const float rs = rsqrtf(row_sum<256>(q, smem) / cols + eps);
    if (threadIdx.x == 0) {
      if (mean_out) mean_out[row] = mu;
      if (rstd_out) rstd_out[row] = rs;
    }
    for (int c = threadIdx.x; c < cols; c += 256) {
      float a = V8<T>::ld1(xr + c);
      if (pre_act == FB_ACT_GELU) a = gelu_f<false>(a);
      const float g = gamma ? gamma[c] : 1.f, b = beta ? beta[c] : 0.f;
      V8<T>::st1(y + row * cols + c, (a - mu) * rs * g + b);
    }
  }
}

// stats = [3][cols] (d_gamma, d_beta, column sum of dx), accumulated into with atomics.
template <typename T>
__global__ void ln_bwd_generic(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ act_grad,
                               const float* __restrict__ gamma, const float* __restrict__ mean,
                               const float* __restrict__ rstd, T* __restrict__ dx, float* __restrict__ stats,
                               long long rows, int cols, int pre_act, int want_colsum) {
  __shared__ float smem[8][8];
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float mu = mean[row], rs = rstd[row];
    float s1 = 0.f, s2 = 0.f;
    for (int c = threadIdx.x; c < cols; c += 256) {
      float a = V8<T>::ld1(x + row * cols + c);
      if (pre_act == FB_ACT_GELU) a = gelu_f<false>(a);
      const float h = (a - mu) * rs;
      const float g = V8<T>::ld1(dy + row * cols + c);
      const float d = g * (gamma ? gamma[c] : 1.f);
      s1 += d;
      s2 += d * h;
      atomicAdd(stats + c, g * h);
      atomicAdd(stats + cols + c, g);
    }
    const float m1 = row_sum<256>(s1, smem) / cols;
    const float m2 = row_sum<256>(s2, smem) / cols;
    for (int c = threadIdx.x; c < cols; c += 256) {
      const float raw = V8<T>::ld1(x + row * cols + c);
      float a = raw, da = 1.f;
      if (pre_act == FB_ACT_GELU) gelu_both<false>(raw, a, da);
      const float h = (a - mu) * rs;
      const float d = V8<T>::ld1(dy + row * cols + c) * (gamma ? gamma[c] : 1.f);
      float o = rs * (d - m1 - h * m2) * da;
      if (act_grad != nullptr) o *= V8<T>::ld1(act_grad + row * cols + c);
      if (want_colsum) atomicAdd(stats + 2 * cols + c, o);
      V8<T>::st1(dx + row * cols + c, o);
    }
  }
}

int sm_count() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return sms;
}

// Fast-path geometry for a row of `cols` elements: threads per row and 8-element vectors per thread.
struct Geo {
  int tpr, k;
};
bool geometry(int cols, Geo* g) {
  if (cols % 8 != 0 || cols > 8192 || cols <= 0) return false;
  const int nvec = cols / 8;
  if (nvec <= 32) *g = {32, 1};
  else if (nvec <= 64) *g = {32, 2};
  else if (nvec <= 128) *g = {128, 1};
  else if (nvec <= 256) *g = {128, 2};
  else if (nvec <= 512) *g = {256, 2};
  else *g = {256, 4};
  return true;
}
// The same for rows of any width: K elements per thread.
bool geometry_any(int cols, Geo* g) {
  if (cols <= 0 || cols > 8192) return false;
  if (cols <= 64) *g = {32, 2};
  else if (cols <= 256) *g = {32, 8};
  else if (cols <= 1024) *g = {128, 8};
  else if (cols <= 2048) *g = {256, 8};
  else if (cols <= 4096) *g = {256, 16};
  else *g = {256, 32};
  return true;
}
#define FB_LN_ANY(g, RUN, WIDER)                     \
  do {                                               \
    if ((g).k == 2) RUN(32, 2);                      \
    else if ((g).tpr == 32) RUN(32, 8);              \
    else if ((g).tpr == 128) RUN(128, 8);            \
    else if ((g).k == 8) RUN(256, 8);                \
    else WIDER;                                      \
  } while (0)

// Where rows of odd width or address are held in registers (any) rather than re-read (generic).  us, generic / any.
// Forward: reading a row three times costs little while it stays in the cache and two blocks' reads overlap; registers
// for 16 or 32 elements a thread leave fewer blocks per SM than the rows want.  fp32, 8192 rows: 257 columns 22.7 / 14.3,
// 1025 26.8 / 23.4, 2049 37 / 52, 4095 70 / 77; 1301 columns: 592 rows 6.3 / 6.3, 1024 6.3 / 8.3, 2048 10.4 / 10.4; 3001:
// 444 rows 8.3 / 6.3, 777 8.3 / 9.7; 7001: 150 rows 10.8 / 10.4, 300 11.5 / 12.6, 2048 29 / 43.  A GELU in front is
// evaluated once instead of three times: 4095 columns, 8192 rows 130 / 84; 7001: 300 rows 16.5 / 15.8, 777 27 / 23, but
// 4097: 300 rows 10.9 / 12.6, 777 16.5 / 18.6.
bool any_fwd(long long rows, int cols, int pre_act) {
  const long long sm = sm_count();
  if (cols > 8192) return false;
  if (pre_act == FB_ACT_GELU) return cols <= 4096 || rows <= sm || rows > 4 * sm;
  if (cols <= 1024) return true;
  if (cols <= 2048) return rows <= 4 * sm || rows > 8 * sm;
  return rows <= (cols <= 4096 ? 3 : 1) * sm;
}
// Backward: for few rows the atomics are cheaper than a second launch; wide rows in registers leave one block per SM.
// bf16, 129 columns: 300 rows 8.3 / 12.4, 777 13.3 / 12.4, 8192 92 / 17; 65: 1024 rows 10.8 / 12.4, 2048 18.5 / 12.4; 1001:
// 300 rows 11.4 / 13.4, 444 13.4 / 13.5, 592 15.5 / 13.5, 8192 122 / 40; 1801, 8192 rows 134 / 120; 2047: 2048 rows 42 / 32,
// 8192 137 / 163; 4097: 2048 rows 64 / 109.  fp32 rows up to 4096: 777 x 2049 25 / 22, 8192 x 2049 151 / 137, 8192 x 4095 194
// / 158; behind a GELU 148 - 251 (the atomics' time varies) / 183 - 205 in that range; 2048 x 4097 70 / 139.
bool any_bwd(long long rows, int cols, bool low) {
  const long long sm = sm_count();
  if (rows <= (cols <= 128 ? 8 : cols <= 256 ? 6 : 3) * sm) return false;
  return cols <= (!low ? 4096 : rows <= 16 * sm ? 2048 : 1792);
}
bool aligned16(const void* a, const void* b, const void* c, const void* d) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
           reinterpret_cast<uintptr_t>(d)) & 15) == 0;
}

int32_t* g_ln_status = nullptr;  // host-mapped status block for the bounded waits of the ring kernels

// FERRUM_LN_RING=0 keeps wide rows on the register-tiled kernels (for A/B measurements).
bool ring_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("FERRUM_LN_RING");
    v = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

template <typename T, int TPR, int K>
void launch_fwd(const T* xp, const float* gamma, const float* beta, T* yp, float* mean, float* rstd, long long rows,
                int cols, float eps, int pre_act, long long nb, cudaStream_t st) {
  const int grid = static_cast<int>(nb < sm_count() * 8LL ? nb : sm_count() * 8LL);
  ln_fwd_kernel<T, TPR, K><<<grid, 256, 0, st>>>(xp, gamma, beta, yp, mean, rstd, rows, cols, eps, pre_act);
}

int env_int(const char* name, int dflt) {
  const char* e = getenv(name);
  return e != nullptr ? atoi(e) : dflt;
}

// Stages per group for slots of `slot_bytes`: as many as fit in `budget` bytes for the two groups of a block,
// at most kMaxRingStages.
int ring_stages(size_t slot_bytes, size_t budget) {
  size_t fit = budget / (2 * slot_bytes);
  static const int forced = env_int("FERRUM_LN_STAGES", 0);  // measurement knob
  if (forced >= 2 && static_cast<size_t>(forced) < fit) fit = forced;
  return static_cast<int>(fit > kMaxRingStages ? kMaxRingStages : fit);
}

// Warp-per-row forward: bf16 rows of 1024 .. 4096 columns without a fused activation (FERRUM_LN_WARP_FWD=0 = off).
template <typename T>
bool launch_fwd_warp(const T*, const float*, const float*, T*, float*, float*, long long, int, float, int,
                     cudaStream_t) {
  return false;
}
template <>
bool launch_fwd_warp<__nv_bfloat16>(const __nv_bfloat16* xp, const float* gamma, const float* beta,
                                    __nv_bfloat16* yp, float* mean, float* rstd, long long rows, int cols, float eps,
                                    int pre_act, cudaStream_t st) {
  static const int enabled = env_int("FERRUM_LN_WARP_FWD", 1);
  if (!enabled || pre_act != FB_ACT_NONE || cols < 1024 || cols > 4096) return false;
  const int k = (cols / 8 + 31) / 32;
  // A block per row while two blocks per SM hold them all: 16 x 4096 6.9 -> 3.5 us, 296 x 2048 4.4 -> 3.2, 296 x 1024
  // 3.0 -> 2.3; at 592 rows the warps are as fast (4096 columns: 7.1 against 7.2 us), at 1184 almost twice as fast.
  if (rows <= 2LL * sm_count()) {
    // It starts beside the tail of the kernel ahead (see ptx::grid_wait).
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(rows));
    cfg.blockDim = dim3(k <= 4 ? 128 : 256);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const auto kernel = k <= 4 ? ln_fwd_warp_kernel<4, 4> : k <= 8 ? ln_fwd_warp_kernel<8, 8> : ln_fwd_warp_kernel<16, 8>;
    cudaLaunchKernelEx(&cfg, kernel, xp, gamma, beta, yp, mean, rstd, rows, cols, eps);
    return true;
  }
  const long long want = (rows + 7) / 8;  // eight warps per block
  const long long cap = static_cast<long long>(sm_count()) * 2;
  const int grid = static_cast<int>(want < cap ? want : cap);
  const size_t smem = static_cast<size_t>(cols) * 8;  // gamma and beta
  if (k <= 4)
    ln_fwd_warp_kernel<4><<<grid, 256, smem, st>>>(xp, gamma, beta, yp, mean, rstd, rows, cols, eps);
  else if (k <= 8)
    ln_fwd_warp_kernel<8><<<grid, 256, smem, st>>>(xp, gamma, beta, yp, mean, rstd, rows, cols, eps);
  else
    ln_fwd_warp_kernel<16><<<grid, 256, smem, st>>>(xp, gamma, beta, yp, mean, rstd, rows, cols, eps);
  return true;
}

// Ring kernel for rows of at least 2 KB and at most 4096 columns; false if it cannot be launched.
template <typename T>
bool launch_fwd_ring(const T* xp, const float* gamma, const float* beta, T* yp, float* mean, float* rstd,
                     long long rows, int cols, float eps, int pre_act, cudaStream_t st) {
  // 2-byte rows run two blocks per SM (register budget of the kernel), so each gets half of the shared memory
  constexpr int kBlocksPerSm = sizeof(T) == 2 ? 2 : 1;
  const int stages = ring_stages(static_cast<size_t>(cols) * sizeof(T), (200u * 1024u) / kBlocksPerSm);
  if (stages < 2) return false;
  const size_t smem = static_cast<size_t>(2 * stages) * cols * sizeof(T);
  static size_t configured = 0;
  if (smem > configured) {
    if (cudaFuncSetAttribute(ln_fwd_ring_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem)) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    configured = smem;
  }
  const long long want = (rows + 1) / 2;  // a block needs two rows to keep both groups busy
  const long long cap = static_cast<long long>(sm_count()) * kBlocksPerSm;
  const int grid = static_cast<int>(want < cap ? (want < 1 ? 1 : want) : cap);
  ln_fwd_ring_kernel<T><<<grid, kRingThreads, smem, st>>>(xp, gamma, beta, yp, mean, rstd, rows, cols, eps, pre_act,
                                                         stages, g_ln_status);
  return true;
}

template <typename T>
int fwd_t(const void* x, const float* gamma, const float* beta, void* y, float* mean, float* rstd, long long rows,
          int cols, float eps, int pre_act, cudaStream_t st) {
  const T* xp = static_cast<const T*>(x);
  T* yp = static_cast<T*>(y);
  Geo g;
  if (geometry(cols, &g) && aligned16(x, y, gamma, beta)) {
    const int nvec = cols / 8;
    if (launch_fwd_warp<T>(xp, gamma, beta, yp, mean, rstd, rows, cols, eps, pre_act, st))
      return static_cast<int>(cudaGetLastError());
    static const int ring_fwd = env_int("FERRUM_LN_RING_FWD", 0);
    if (ring_fwd && ring_enabled() && static_cast<size_t>(cols) * sizeof(T) >= 2048 && nvec <= 2 * kGroupThreads &&
        launch_fwd_ring<T>(xp, gamma, beta, yp, mean, rstd, rows, cols, eps, pre_act, st))
      return static_cast<int>(cudaGetLastError());
    const long long rpb = 256 / g.tpr;
    const long long nb = (rows + rpb - 1) / rpb;
#define FB_LN_FWD(TPR, K) \
  launch_fwd<T, TPR, K>(xp, gamma, beta, yp, mean, rstd, rows, cols, eps, pre_act, nb, st)
    if (g.tpr == 32 && g.k == 1) FB_LN_FWD(32, 1);
    else if (g.tpr == 32) FB_LN_FWD(32, 2);
    else if (g.tpr == 128 && g.k == 1) FB_LN_FWD(128, 1);
    else if (g.tpr == 128) FB_LN_FWD(128, 2);
    else if (g.k == 2) FB_LN_FWD(256, 2);
    else FB_LN_FWD(256, 4);
#undef FB_LN_FWD
  } else if (any_fwd(rows, cols, pre_act) && geometry_any(cols, &g)) {
    const long long nb = (rows + 256 / g.tpr - 1) / (256 / g.tpr);
    const int grid = static_cast<int>(nb < sm_count() * 8LL ? nb : sm_count() * 8LL);
#define FB_LN_FWD(TPR, K) \
  ln_fwd_any_kernel<T, TPR, K><<<grid, 256, 0, st>>>(xp, gamma, beta, yp, mean, rstd, rows, cols, eps, pre_act)
    FB_LN_ANY(g, FB_LN_FWD, if (g.k == 16) FB_LN_FWD(256, 16); else FB_LN_FWD(256, 32));
#undef FB_LN_FWD
  } else {
    const int grid = static_cast<int>(rows < sm_count() * 8LL ? rows : sm_count() * 8LL);
    ln_fwd_generic<T><<<grid, 256, 0, st>>>(xp, gamma, beta, yp, mean, rstd, rows, cols, eps, pre_act);
  }
  return static_cast<int>(cudaGetLastError());
}

template <typename R>
int add_fwd_t(const float* x, const R* r, const float* gamma, const float* beta, float* sum, float* y, float* mean,
              float* rstd, long long rows, int cols, float eps, cudaStream_t st) {
  Geo g;
  if (!geometry(cols, &g) || !aligned16(x, r, gamma, beta) || !aligned16(sum, y, nullptr, nullptr)) return -2;
  const long long nb = (rows + 256 / g.tpr - 1) / (256 / g.tpr);
  const int grid = static_cast<int>(nb < sm_count() * 8LL ? nb : sm_count() * 8LL);
#define FB_LN_ADD(TPR, K) \
  ln_add_fwd_kernel<R, TPR, K><<<grid, 256, 0, st>>>(x, r, gamma, beta, sum, y, mean, rstd, rows, cols, eps)
  if (g.tpr == 32 && g.k == 1) FB_LN_ADD(32, 1);
  else if (g.tpr == 32) FB_LN_ADD(32, 2);
  else if (g.tpr == 128 && g.k == 1) FB_LN_ADD(128, 1);
  else if (g.tpr == 128) FB_LN_ADD(128, 2);
  else if (g.k == 2) FB_LN_ADD(256, 2);
  else FB_LN_ADD(256, 4);
#undef FB_LN_ADD
  return static_cast<int>(cudaGetLastError());
}

template <typename T>
bool launch_wide(const T*, const T*, const T*, const float*, const float*, const float*, T*, float*, long long, int,
                 int, int, float*, cudaStream_t) {
  return false;
}
// bf16 rows of 2 KB .. 8 KB with no activation to re-evaluate: the ring kernel, one block per SM.
template <>
bool launch_wide<__nv_bfloat16>(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* ag,
                                const float* gamma, const float* mean, const float* rstd, __nv_bfloat16* dx,
                                float* partial, long long rows, int cols, int blocks, int want_colsum, float* clear,
                                cudaStream_t st) {
  const int stages = ring_stages(static_cast<size_t>(cols) * 2 * (ag != nullptr ? 3 : 2), 200u * 1024u);
  if (stages < 2) return false;
  const size_t smem = static_cast<size_t>(2 * stages) * (ag != nullptr ? 3 : 2) * cols * 2;
  static size_t configured = 0;
  if (smem > configured) {
    if (cudaFuncSetAttribute(ln_bwd_ring_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem)) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    configured = smem;
  }
  ln_bwd_ring_kernel<<<blocks, kRingThreads, smem, st>>>(dy, x, ag, gamma, mean, rstd, dx, partial, rows, cols,
                                                         want_colsum, stages, g_ln_status, clear);
  return true;
}

template <typename T>
int bwd_t(const void* dy, const void* x, const void* act_grad, const float* gamma, const float* mean,
          const float* rstd, void* dx, __nv_bfloat16* dx_low, float* partial, float* stats, long long rows, int cols,
          int pre_act, int nblk, int flags, cudaStream_t st) {
  const int want_colsum = flags & 1;
  float* clear = (flags & 2) != 0 ? stats : nullptr;
  const T* dyp = static_cast<const T*>(dy);
  const T* xp = static_cast<const T*>(x);
  const T* agp = static_cast<const T*>(act_grad);
  T* dxp = static_cast<T*>(dx);
  Geo g;
  const bool fast = nblk > 0 && partial != nullptr && geometry(cols, &g) && aligned16(dy, x, dx, gamma) &&
                    aligned16(partial, stats, act_grad, dx_low);
  if (dx_low != nullptr && !fast) return -2;
  Geo any;
  if (fast || (nblk > 0 && partial != nullptr && any_bwd(rows, cols, sizeof(T) == 2) && geometry_any(cols, &any))) {
    int used = nblk;
    const int nvec = cols / 8;
    const int wide_blocks = nblk / 2 < sm_count() ? nblk / 2 : sm_count();  // two rows of partial[] per block
    if (fast && dx_low == nullptr && ring_enabled() && pre_act == FB_ACT_NONE && cols * 2 >= 2048 && nvec <= 2 * kGroupThreads &&
        wide_blocks >= 1 &&
        launch_wide<T>(dyp, xp, agp, gamma, mean, rstd, dxp, partial, rows, cols, wide_blocks, want_colsum, clear, st)) {
      used = 2 * wide_blocks;
    } else if (!fast) {
#define FB_LN_BWD(TPR, K) \
  ln_bwd_any_kernel<T, TPR, K><<<nblk, 256, 0, st>>>(dyp, xp, agp, gamma, mean, rstd, dxp, partial, rows, cols, pre_act, \
                                                     want_colsum, clear)
      FB_LN_ANY(any, FB_LN_BWD, if constexpr (sizeof(T) == 4) FB_LN_BWD(256, 16));
#undef FB_LN_BWD
    } else {
      const auto run = [&](auto plain, auto low) {
        (dx_low != nullptr ? low : plain)<<<nblk, 256, 0, st>>>(dyp, xp, agp, gamma, mean, rstd, dxp, dx_low, partial, rows,
                                                                cols, pre_act, want_colsum, clear);
      };
#define FB_LN_BWD(TPR, K) run(ln_bwd_kernel<T, TPR, K, K == 4>, ln_bwd_kernel<T, TPR, K, K == 4 || sizeof(T) == 4>)
    if (g.tpr == 32 && g.k == 1) FB_LN_BWD(32, 1);
    else if (g.tpr == 32) FB_LN_BWD(32, 2);
    else if (g.tpr == 128 && g.k == 1) FB_LN_BWD(128, 1);
    else if (g.tpr == 128) FB_LN_BWD(128, 2);
    else if (g.k == 2) FB_LN_BWD(256, 2);
    else FB_LN_BWD(256, 4);
#undef FB_LN_BWD
    }
    const int ncols = 3 * cols;
    const int col_blocks = (ncols + 127) / 128;
    int row_blocks = (sm_count() * 2 + col_blocks - 1) / col_blocks;
    const int max_rb = (used + 15) / 16;
    if (row_blocks > max_rb) row_blocks = max_rb;
    if (row_blocks < 1) row_blocks = 1;
    const int rpb = (used + row_blocks - 1) / row_blocks;
    const auto fold = ncols % 4 == 0 && aligned16(partial, nullptr, nullptr, nullptr) ? ln_fold_kernel<true> : ln_fold_kernel<false>;
    fold<<<dim3(col_blocks, row_blocks), 256, 0, st>>>(partial, stats, used, ncols, rpb);
  } else {
    if (clear != nullptr) {
      const cudaError_t e = cudaMemsetAsync(stats, 0, 3 * static_cast<size_t>(cols) * sizeof(float), st);
      if (e != cudaSuccess) return static_cast<int>(e);
    }
    const int grid = static_cast<int>(rows < sm_count() * 4LL ? rows : sm_count() * 4LL);
    ln_bwd_generic<T><<<grid, 256, 0, st>>>(dyp, xp, agp, gamma, mean, rstd, dxp, stats, rows, cols, pre_act,
                                            want_colsum);
  }
  return static_cast<int>(cudaGetLastError());
}

}  // namespace
}  // namespace fb

using namespace fb;

// Status block (host-mapped, see common/status.h) that the bounded waits of the wide-row kernels report to.
extern "C" void fb_layernorm_set_status(int32_t* status) { g_ln_status = status; }

// Number of blocks (= rows of `partial`, each 3 * cols floats) the backward uses; 0 means that the generic path runs and
// no partial buffer is needed.
extern "C" int fb_layernorm_bwd_blocks(long long rows, int cols) {
  Geo g;
  if (!geometry(cols, &g) && !(any_bwd(rows, cols, false) && geometry_any(cols, &g))) return 0;
  const long long rpb = 256 / g.tpr;
  const long long nb = (rows + rpb - 1) / rpb;
  // Three blocks per SM where a thread holds one vector of a row: loads in flight, not registers, are what is short.
  const long long cap = static_cast<long long>(sm_count()) * (cols % 8 == 0 && g.k == 1 ? 3 : 2);
  return static_cast<int>(nb < cap ? nb : cap);
}

extern "C" int fb_layernorm_fwd(const void* x, const float* gamma, const float* beta, void* y, float* mean,
                                float* rstd, long long rows, int cols, float eps, int pre_act, int dtype,
                                cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return 0;
  if (dtype == FB_DT_F32) return fwd_t<float>(x, gamma, beta, y, mean, rstd, rows, cols, eps, pre_act, stream);
  if (dtype == FB_DT_BF16)
    return fwd_t<__nv_bfloat16>(x, gamma, beta, y, mean, rstd, rows, cols, eps, pre_act, stream);
  return -1;
}

// stats = [3][cols] fp32: d_gamma, d_beta and the column sum of dx.  All three are ACCUMULATED into (zero the buffer for a
// fresh gradient), or written where want_colsum has the bit 2; the column sum is produced only where it has the bit 1.
// act_grad (optional, dtype of x): x then holds act(z) of an activation applied before the normalisation and
// act_grad its derivative act'(z); dx is the gradient of z.  (pre_act instead re-evaluates a GELU from z.)
extern "C" int fb_layernorm_bwd(const void* dy, const void* x, const void* act_grad, const float* gamma,
                                const float* mean, const float* rstd, void* dx, float* partial, float* stats,
                                long long rows, int cols, int pre_act, int dtype, int nblk, int want_colsum,
                                cudaStream_t stream) {
  if (cols <= 0) return 0;
  if (rows <= 0)  // empty sums
    return (want_colsum & 2) == 0 || stats == nullptr
               ? 0
               : static_cast<int>(cudaMemsetAsync(stats, 0, 3 * static_cast<size_t>(cols) * sizeof(float), stream));
  if (stats == nullptr) return -1;
  if (act_grad != nullptr && pre_act != FB_ACT_NONE) return -1;
  if (dtype == FB_DT_F32)
    return bwd_t<float>(dy, x, act_grad, gamma, mean, rstd, dx, nullptr, partial, stats, rows, cols, pre_act, nblk,
                        want_colsum, stream);
  if (dtype == FB_DT_BF16)
    return bwd_t<__nv_bfloat16>(dy, x, act_grad, gamma, mean, rstd, dx, nullptr, partial, stats, rows, cols, pre_act, nblk,
                                want_colsum, stream);
  return -1;
}

// norm(x + r) of fp32 x and r of r_dtype; sum (optional) = x + r.  -2, and nothing is launched: widths or addresses that
// are not made of whole 16-byte pieces, more than 8192 columns.
extern "C" int fb_add_layernorm_fwd(const float* x, const void* r, const float* gamma, const float* beta, float* sum,
                                    float* y, float* mean, float* rstd, long long rows, int cols, float eps, int r_dtype,
                                    cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return 0;
  if (mean == nullptr || rstd == nullptr) return -1;
  if (r_dtype == FB_DT_F32)
    return add_fwd_t<float>(x, static_cast<const float*>(r), gamma, beta, sum, y, mean, rstd, rows, cols, eps, stream);
  if (r_dtype == FB_DT_BF16)
    return add_fwd_t<__nv_bfloat16>(x, static_cast<const __nv_bfloat16*>(r), gamma, beta, sum, y, mean, rstd, rows, cols,
                                    eps, stream);
  return -1;
}

// fb_layernorm_bwd of fp32 rows, whose dx also goes to dx_low (optional) in bf16; stats are written.
extern "C" int fb_add_layernorm_bwd(const float* dy, const float* sum, const float* gamma, const float* mean,
                                    const float* rstd, float* dx, void* dx_low, float* partial, float* stats,
                                    long long rows, int cols, int nblk, cudaStream_t stream) {
  if (cols <= 0) return 0;
  if (stats == nullptr) return -1;
  if (rows <= 0) return static_cast<int>(cudaMemsetAsync(stats, 0, 3 * static_cast<size_t>(cols) * sizeof(float), stream));
  return bwd_t<float>(dy, sum, nullptr, gamma, mean, rstd, dx, static_cast<__nv_bfloat16*>(dx_low), partial, stats, rows,
                      cols, FB_ACT_NONE, nblk, 2, stream);
}
