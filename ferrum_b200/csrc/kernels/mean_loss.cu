// Mean losses that end in one scalar: cross-entropy of logits, NLL of log-probabilities, and the elementwise losses.
//
// A forward pass is a sum over the whole input, so many blocks have to meet in one number.  Small inputs run as ONE
// cluster of eight blocks that adds its partial sums through distributed shared memory: one launch, no workspace to
// clear, no atomics, the same order of additions every time.  Larger inputs need the whole chip for bandwidth: the
// blocks leave one partial sum each and a one-block kernel adds them in order.  The line between the two lies where
// eight SMs stream the input in about the time that the second launch takes (256 K elements).
//
// The cross-entropy writes the logit gradient of a unit loss in the forward pass, from the exponentials it has at hand,
// and the backward pass scales it by the incoming gradient: the logits are the caller's again once the loss is known.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>

#include "../common/status.h"
#include "../include/ferrum_kernels.h"

namespace fb {
namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 256;
constexpr int kCluster = 8;
constexpr long long kClusterElems = 256 * 1024;
constexpr int kClusterTrips = 3;
constexpr int kMaxPartials = 1184;  // 8 blocks per SM on 148 SMs

__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ void put(float* p, float v) { *p = v; }
__device__ __forceinline__ void put(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int TPR, bool IS_MAX>
__device__ __forceinline__ float group_reduce(float v, float* smem) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float u = __shfl_xor_sync(0xffffffffu, v, o);
    v = IS_MAX ? fmaxf(v, u) : v + u;
  }
  if (TPR == 32) return v;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  float t = IS_MAX ? -FLT_MAX : 0.f;
#pragma unroll
  for (int w = 0; w < TPR / 32; ++w) t = IS_MAX ? fmaxf(t, smem[w]) : t + smem[w];
  return t;
}

// Adds `v` over the block (and the cluster) and stores the result: partial sum of the block, or scale * total.
template <bool kClustered>
__device__ __forceinline__ void finish(float v, float scale, float* loss, float* partial) {
  __shared__ float part[kThreads / 32];
  __shared__ float block_total;
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) t += part[w];
    block_total = t;
    if (!kClustered) partial[blockIdx.x] = t;
  }
  if constexpr (kClustered) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (cluster.block_rank() == 0 && threadIdx.x == 0) {
      float t = 0.f;
      for (int r = 0; r < kCluster; ++r) t += *cluster.map_shared_rank(&block_total, r);
      *loss = t * scale;
    }
    cluster.sync();
  }
}

__global__ void __launch_bounds__(kThreads) add_partials_kernel(const float* __restrict__ partial, int n, float scale,
                                                                float* __restrict__ loss) {
  __shared__ float part[kThreads / 32];
  float v = 0.f;
  for (int i = threadIdx.x; i < n; i += kThreads) v += partial[i];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) t += part[w];
    *loss = t * scale;
  }
}

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 t = __bfloat1622float2(h[e]);
    f[2 * e] = t.x;
    f[2 * e + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 raw;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
  *reinterpret_cast<uint4*>(p) = raw;
}

// Rows of 264 .. 4096 bf16 logits (multiples of 8, 16-byte aligned): a warp owns a row and keeps it in registers (K
// vectors of 8 per lane), so the row is read once and both reductions are warp shuffles.
template <int K, bool kClustered>
__global__ void __launch_bounds__(kThreads, K <= 4 ? 4 : (K <= 8 ? 2 : 1))
ce_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x, const long long* __restrict__ labels,
                   __nv_bfloat16* __restrict__ dx, float* __restrict__ loss, float* __restrict__ partial, long long rows,
                   int cols, float scale, int32_t* bstatus) {
  const int lane = threadIdx.x & 31;
  const int nvec = cols >> 3;
  const long long nwarps = static_cast<long long>(gridDim.x) * (kThreads / 32);
  float acc = 0.f;
  for (long long row = static_cast<long long>(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5); row < rows;
       row += nwarps) {
    const __nv_bfloat16* xr = x + row * cols;
    float v[K][8];
    float m = -FLT_MAX;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int vi = lane + 32 * k;
      if (vi < nvec) {
        load8(xr + vi * 8, v[k]);
#pragma unroll
        for (int e = 0; e < 8; ++e) m = fmaxf(m, v[k][e]);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[k][e] = -FLT_MAX;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        v[k][e] = __expf(v[k][e] - m);  // padded lanes: exp(-huge) = 0
        s += v[k][e];
      }
    s = warp_sum(s);
    const long long lab = labels[row];
    const bool valid = lab >= 0 && lab < cols;  // out-of-range labels contribute nothing
    if (lane == 0) {
      if (!valid) (void)FB_INDEX_OK(bstatus, 41, lab, cols);
      if (valid) acc += m + logf(s) - __bfloat162float(xr[lab]);
    }
    if (dx != nullptr) {
      const float inv = valid ? scale / s : 0.f;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int vi = lane + 32 * k;
        if (vi >= nvec) continue;
        float d[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          d[e] = v[k][e] * inv;
          if (valid && vi * 8 + e == lab) d[e] -= scale;
        }
        store8(dx + row * cols + vi * 8, d);
      }
    }
  }
  finish<kClustered>(acc, scale, loss, partial);
}

// Any other row: TPR threads per row, the row is read again from L1 for the sum and for the gradient.
template <typename T, int TPR, bool kClustered>
__global__ void __launch_bounds__(kThreads)
ce_fwd_kernel(const T* __restrict__ x, const long long* __restrict__ labels, T* __restrict__ dx,
              float* __restrict__ loss, float* __restrict__ partial, long long rows, int cols, float scale,
              int32_t* bstatus) {
  __shared__ float smem[kThreads / 32];
  constexpr int kRows = kThreads / TPR;
  const int sub = threadIdx.x / TPR, t = threadIdx.x % TPR;
  float acc = 0.f;
  for (long long row0 = static_cast<long long>(blockIdx.x) * kRows; row0 < rows;
       row0 += static_cast<long long>(gridDim.x) * kRows) {
    const long long row = row0 + sub;
    const bool live = row < rows;
    const T* xr = x + (live ? row : 0) * cols;
    float m = -FLT_MAX, s = 0.f;
    if (live)
      for (int c = t; c < cols; c += TPR) m = fmaxf(m, to_f(xr[c]));
    m = group_reduce<TPR, true>(m, smem);
    if (live)
      for (int c = t; c < cols; c += TPR) s += expf(to_f(xr[c]) - m);
    s = group_reduce<TPR, false>(s, smem);
    const long long lab = live ? labels[row] : -1;
    const bool valid = lab >= 0 && lab < cols;
    if (live && t == 0) {
      if (!valid) (void)FB_INDEX_OK(bstatus, 41, lab, cols);
      if (valid) acc += m + logf(s) - to_f(xr[lab]);
    }
    if (live && dx != nullptr) {
      const float inv = 1.f / s;
      for (int c = t; c < cols; c += TPR) {
        float f = expf(to_f(xr[c]) - m) * inv;
        if (c == lab) f -= 1.f;
        put(dx + row * cols + c, valid ? f * scale : 0.f);
      }
    }
  }
  finish<kClustered>(acc, scale, loss, partial);
}

template <typename T, bool kClustered>
__global__ void __launch_bounds__(kThreads)
nll_fwd_kernel(const T* __restrict__ lp, const long long* __restrict__ target, float* __restrict__ loss,
               float* __restrict__ partial, long long rows, int cols, float scale, int32_t* status) {
  float acc = 0.f;
  const long long stride = static_cast<long long>(gridDim.x) * kThreads;
  for (long long r = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x; r < rows; r += stride) {
    const long long t = target[r];
    // a class outside the range is an error: in the status block (every build), and the loss shows it
    acc += check_index(status, 42, t, cols) ? to_f(lp[r * cols + t]) : __int_as_float(0x7fffffff);
  }
  finish<kClustered>(acc, scale, loss, partial);
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
nll_bwd_kernel(const long long* __restrict__ target, const float* __restrict__ gout, T* __restrict__ dx, long long n,
               int cols, float scale) {
  const float g = gout[0] * scale;
  const long long stride = static_cast<long long>(gridDim.x) * kThreads;
  for (long long i = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x; i < n; i += stride) {
    const long long r = i / cols;
    put(dx + i, i - r * cols == target[r] ? g : 0.f);
  }
}

__device__ __forceinline__ float loss_of(float p, float t, int kind) {
  const float d = p - t;
  switch (kind) {
    case FB_LOSS_MSE: return d * d;
    case FB_LOSS_BCE: {
      const float eps = 1e-7f, pc = p + eps, q = (1.f + eps) - pc;
      return -(t * logf(pc) + (1.f - t) * logf(q));
    }
    case FB_LOSS_L1: return fabsf(d);
    default: {
      const float a = fabsf(d);
      return a < 1.f ? 0.5f * d * d : a - 0.5f;
    }
  }
}

template <bool kClustered>
__global__ void __launch_bounds__(kThreads)
elem_loss_kernel(const float* __restrict__ p, const float* __restrict__ t, float* __restrict__ loss,
                 float* __restrict__ partial, long long n, int kind, float scale) {
  float acc = 0.f;
  const long long stride = static_cast<long long>(gridDim.x) * kThreads;
  const long long tid = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x;
  const bool al = ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(t)) & 15) == 0;
  const long long n4 = al ? n >> 2 : 0;
#pragma unroll 4
  for (long long i = tid; i < n4; i += stride) {
    const float4 a = reinterpret_cast<const float4*>(p)[i], b = reinterpret_cast<const float4*>(t)[i];
    acc += loss_of(a.x, b.x, kind) + loss_of(a.y, b.y, kind) + loss_of(a.z, b.z, kind) + loss_of(a.w, b.w, kind);
  }
  for (long long i = (n4 << 2) + tid; i < n; i += stride) acc += loss_of(p[i], t[i], kind);
  finish<kClustered>(acc, scale, loss, partial);
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

int wide_grid(long long blocks) {
  long long cap = static_cast<long long>(sm_count()) * 8;
  if (cap > kMaxPartials) cap = kMaxPartials;
  return static_cast<int>(blocks < cap ? (blocks < 1 ? 1 : blocks) : cap);
}

// Launches the one-cluster form of a kernel for small inputs, else the wide form followed by the final addition.
template <typename... P, typename... A>
int run_mean(void (*clustered)(P...), void (*wide)(P...), bool small, long long blocks, float* loss, float* partial,
             float scale, cudaStream_t st, A... args) {
  if (small) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kCluster);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kCluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return static_cast<int>(cudaLaunchKernelEx(&cfg, clustered, args...));
  }
  const int grid = wide_grid(blocks);
  wide<<<grid, kThreads, 0, st>>>(args...);
  add_partials_kernel<<<1, kThreads, 0, st>>>(partial, grid, scale, loss);
  return static_cast<int>(cudaGetLastError());
}

bool vec_ok(const void* a, const void* b, int cols, size_t elem) {
  return cols % static_cast<int>(16 / elem) == 0 &&
         ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
}
// Rows that the register-resident warp kernel takes.
bool warp_row(const void* x, const void* dx, int cols) { return cols >= 264 && cols <= 4096 && vec_ok(x, dx, cols, 2); }

// A row of a cross-entropy is a chain of loads, reductions and exponentials, 1.2 us of a warp: the cluster's eight blocks
// take at most three rounds of them, beyond that the whole chip and a second launch are faster or as fast.  One cluster /
// whole chip, us: 37 classes bf16 (eight rows per block) 193 rows 8.2 / 8.2, 384 11.3 / 7.2, 777 20.4 / 8.2; 1000 classes
// fp32 (a row per block) 24 rows 8.4 / 8, 25 10.3 / 8.2, 193 43 / 7.2.
bool few_rows(long long elems, long long blocks) { return elems <= kClusterElems && blocks <= kClusterTrips * kCluster; }

template <typename T>
int ce_fwd(const void* x, const long long* labels, void* dlogits, float* loss, float* partial, long long rows, int cols,
           float scale, cudaStream_t st) {
  T* dx = static_cast<T*>(dlogits);
  if constexpr (sizeof(T) == 2) {
    if (warp_row(x, dx, cols)) {
      const int k = (cols / 8 + 31) / 32;
#define FB_CE_WARP(K)                                                                                                  \
  return run_mean(ce_fwd_warp_kernel<K, true>, ce_fwd_warp_kernel<K, false>, few_rows(rows * cols, (rows + 7) / 8),     \
                  (rows + 7) / 8, loss, partial, scale, st, static_cast<const __nv_bfloat16*>(x), labels, dx, loss, partial, rows, cols, scale,      \
                  bounds_status_ref())
      if (k <= 4) FB_CE_WARP(4);
      if (k <= 8) FB_CE_WARP(8);
      FB_CE_WARP(16);
#undef FB_CE_WARP
    }
  }
  if (cols <= 512)
    return run_mean(ce_fwd_kernel<T, 32, true>, ce_fwd_kernel<T, 32, false>, few_rows(rows * cols, (rows + 7) / 8),
                    (rows + 7) / 8, loss, partial, scale, st, static_cast<const T*>(x), labels, dx, loss, partial, rows,
                    cols, scale, bounds_status_ref());
  return run_mean(ce_fwd_kernel<T, 256, true>, ce_fwd_kernel<T, 256, false>, few_rows(rows * cols, rows), rows, loss,
                  partial, scale, st, static_cast<const T*>(x), labels, dx, loss, partial, rows, cols, scale,
                  bounds_status_ref());
}

}  // namespace
}  // namespace fb

using namespace fb;

extern "C" long long fb_mean_loss_workspace(long long) { return kMaxPartials; }

extern "C" int fb_ce_fwd(const void* logits, const long long* labels, void* dlogits, float* loss, float* workspace,
                         long long rows, int cols, float scale, int dtype, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return -1;  // no mean over nothing: `loss` stays unwritten
  if (dtype == FB_DT_F32) return ce_fwd<float>(logits, labels, dlogits, loss, workspace, rows, cols, scale, stream);
  if (dtype == FB_DT_BF16)
    return ce_fwd<__nv_bfloat16>(logits, labels, dlogits, loss, workspace, rows, cols, scale, stream);
  return -1;
}

extern "C" int fb_nll_fwd(const void* log_probs, const long long* target, float* loss, float* workspace, long long rows,
                          int cols, float scale, int dtype, int32_t* status, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return -1;  // no mean over nothing: `loss` stays unwritten
  const long long blocks = (rows + kThreads - 1) / kThreads;
  if (dtype == FB_DT_F32)
    return run_mean(nll_fwd_kernel<float, true>, nll_fwd_kernel<float, false>, rows <= kClusterElems, blocks, loss, workspace,
                    scale, stream, static_cast<const float*>(log_probs), target, loss, workspace, rows, cols, scale, status);
  if (dtype == FB_DT_BF16)
    return run_mean(nll_fwd_kernel<__nv_bfloat16, true>, nll_fwd_kernel<__nv_bfloat16, false>, rows <= kClusterElems, blocks,
                    loss, workspace, scale, stream, static_cast<const __nv_bfloat16*>(log_probs), target, loss, workspace,
                    rows, cols, scale, status);
  return -1;
}

extern "C" int fb_nll_bwd(const long long* target, const float* gout, void* dlog_probs, long long rows, int cols,
                          float scale, int dtype, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return 0;
  const long long n = rows * cols;
  long long nb = (n + kThreads - 1) / kThreads;
  const long long cap = static_cast<long long>(sm_count()) * 8;
  if (nb > cap) nb = cap;
  if (dtype == FB_DT_F32)
    nll_bwd_kernel<float><<<static_cast<int>(nb), kThreads, 0, stream>>>(target, gout, static_cast<float*>(dlog_probs),
                                                                        n, cols, scale);
  else if (dtype == FB_DT_BF16)
    nll_bwd_kernel<__nv_bfloat16><<<static_cast<int>(nb), kThreads, 0, stream>>>(
        target, gout, static_cast<__nv_bfloat16*>(dlog_probs), n, cols, scale);
  else
    return -1;
  return static_cast<int>(cudaGetLastError());
}

extern "C" int fb_loss_mean_fwd(const float* pred, const float* target, float* loss, float* workspace, long long n,
                                int kind, float scale, cudaStream_t stream) {
  if (n <= 0) return -1;
  return run_mean(elem_loss_kernel<true>, elem_loss_kernel<false>, n <= kClusterElems,
                  (n + 4 * kThreads - 1) / (4 * kThreads), loss, workspace, scale, stream, pred, target, loss, workspace, n, kind, scale);
}
