// Column sums of a matrix whose rows are divided among the blocks of a cluster (along y): every block's sums meet in the
// first one through distributed shared memory, in the order of the blocks.  No atomics, so no result to clear first: one launch
// instead of two.  With a fill and atomics / so, us, one after another in a stream: 128 x 256 bf16 6.1 / 5.2 (as nodes of a graph
// 6.0 / 3.4), 1024 x 1000 6.3 / 6.3 (6.3 / 4.2), 2048 x 4096 9.3 / 7.3, 8192 x 1024 fp32 out of memory 14.4 / 10.3; ReLU gradient
// and column sums of 8192 x 4096 bf16 49 as three launches, 37 as one.
#pragma once
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace fb {
namespace {

// Every thread of every block: part[n] in shared memory, complete but not yet synchronised.  write(i, sum) runs in the first
// block; no block leaves before its sums have been read.
template <class F>
__device__ __forceinline__ void cluster_sums(const float* part, int n, F&& write) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int blocks = static_cast<int>(cluster.num_blocks());
  if (blocks == 1) {
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) write(i, part[i]);
    return;
  }
  cluster.sync();
  if (cluster.block_rank() == 0) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      float v[8], s = 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < blocks) v[r] = cluster.map_shared_rank(part, r)[i];
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < blocks) s += v[r];
      write(i, s);
    }
  }
  cluster.sync();
}

inline int column_sms() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}

constexpr int kColumnThreads = 512;

// A launch with clusters of grid.y blocks (at most 8).
template <class... P, class... A>
int launch_column_cluster(void (*kernel)(P...), dim3 grid, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kColumnThreads);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = at[0].val.clusterDim.z = 1;
  at[0].val.clusterDim.y = grid.y;
  cfg.attrs = at;
  cfg.numAttrs = grid.y > 1 ? 1 : 0;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, args...));
}

template <typename T>
__device__ __forceinline__ void unpack16(const uint4& u, float (&v)[16 / sizeof(T)]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (sizeof(T) == 4) {
      v[i] = __uint_as_float(w[i]);
    } else {  // bf16 -> fp32 is a 16-bit shift
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
}

// The matrix as it is.
template <typename T>
struct PlainRows {
  static constexpr int kV = 16 / sizeof(T), kU = 8, kPerSm = 2;
  using Raw = uint4;
  const T* x;
  __host__ __device__ bool aligned() const { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; }
  __device__ Raw fetch(long long at) const { return *reinterpret_cast<const uint4*>(x + at); }
  __device__ void use(const Raw& r, long long, float (&v)[kV]) const { unpack16<T>(r, v); }
  __device__ float one(long long at) const { return static_cast<float>(x[at]); }
};

// A block sums L lanes x 16 bytes of columns over its rows, 512 / L of them at a time with Rows::kU loads each in flight: there
// are hardly more blocks than SMs, so a block of whole pieces keeps 64 KB on their way.
// Two blocks to an SM: a grid is up to twice the SMs, and with one of them at a time (90 registers for a gradient with four
// loads of each operand) its second half took a turn of its own.  ReLU gradient and sums, bf16, us, two launches / one block /
// two: 8192 x 2048 20.5 / 28.4 / 14.5, 16384 x 1024 21.0 / 27.1 / 21.8, 2048 x 2048 7.8 / 11.1 / 6.2.
template <class Rows, int L>
__global__ void __launch_bounds__(kColumnThreads, Rows::kPerSm)
colsum_cluster_kernel(const Rows m, float* __restrict__ out, long long rows, long long cols, long long rows_per_block,
                      int accumulate) {
  constexpr int kV = Rows::kV, kU = Rows::kU, kR = kColumnThreads / L, kCols = L * kV;
  __shared__ float warps[kColumnThreads / 32][kCols], part[kCols];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = threadIdx.x % L;
  const long long c0 = static_cast<long long>(blockIdx.x) * kCols + l * kV;
  const long long r_lo = static_cast<long long>(blockIdx.y) * rows_per_block, r_hi = min(rows, r_lo + rows_per_block);
  float acc[kV];
#pragma unroll
  for (int i = 0; i < kV; ++i) acc[i] = 0.f;
  if (cols % kV == 0 && m.aligned()) {
    if (c0 < cols) {
      for (long long r = r_lo + threadIdx.x / L; r < r_hi; r += kR * kU) {
        typename Rows::Raw raw[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u)
          if (r + u * kR < r_hi) raw[u] = m.fetch((r + u * kR) * cols + c0);
#pragma unroll
        for (int u = 0; u < kU; ++u)
          if (r + u * kR < r_hi) {
            float v[kV];
            m.use(raw[u], (r + u * kR) * cols + c0, v);
#pragma unroll
            for (int i = 0; i < kV; ++i) acc[i] += v[i];
          }
      }
    }
  } else {
    for (long long r = r_lo + threadIdx.x / L; r < r_hi; r += kR)
#pragma unroll
      for (int i = 0; i < kV; ++i)
        if (c0 + i < cols) acc[i] += m.one(r * cols + c0 + i);
  }
#pragma unroll
  for (int d = L; d < 32; d *= 2)
#pragma unroll
    for (int i = 0; i < kV; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], d);
  if (lane < L) {
#pragma unroll
    for (int i = 0; i < kV; ++i) warps[warp][l * kV + i] = acc[i];
  }
  __syncthreads();
  if (threadIdx.x < kCols) {
    const int t = threadIdx.x;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kColumnThreads / 32; ++w) s += warps[w][t];
    part[t] = s;
  }
  cluster_sums(part, kCols, [&](int i, float s) {
    const long long c = static_cast<long long>(blockIdx.x) * kCols + i;
    if (c < cols) out[c] = accumulate ? out[c] + s : s;
  });
}

struct ColumnPlan {
  int lanes, split;  // 16-byte pieces of a row to a block, blocks to a column range
  long long ranges;
};
inline ColumnPlan column_plan(long long rows, long long cols, int v) {  // v: elements of 16 bytes
  // 128 bytes of a row to a block, or 64 or 32 where that would leave a third of the chip without one (memory is read by
  // lines: 8192 x 1024 bf16 9.7 us with 32 bytes, 7.6 with 128).
  ColumnPlan p{8, 1, 0};
  while (p.lanes > 2 && (cols + p.lanes * v - 1) / (p.lanes * v) * 8 * 3 < column_sms() * 2) p.lanes /= 2;
  p.ranges = (cols + p.lanes * v - 1) / (p.lanes * v);
  // As many blocks to a range as give every SM one: with eight to each of 64 ranges they took turns (512 x 4096 bf16 7.5 us).
  while (p.split < 8 && p.ranges * p.split < column_sms() && rows >= p.split * 64) p.split *= 2;
  return p;
}
// Whether one launch of clusters is faster than the sums in a cleared buffer (size: bytes of an element; grad: behind an
// activation's gradient, then than a pass for each).  It saves a launch, or two; but a column range has eight blocks at most,
// with fewer loads on their way than the four smaller ones to every SM there, so few blocks with much to read are slower.
// us, otherwise / in one launch, one after another in a stream:
//  - Never more than 4 MB in ranges of 32 bytes that leave SMs without a block.
//  - Whole pieces: 96 KB to a block pay, and more where the ranges are wide (fp32 32768 x 1024 36 / 26, with a gradient bf16
//    8192 x 2048 25.6 / 16.5).  Not where they are narrow (with a gradient bf16 32768 x 64 12.4 / 14.5, 32768 x 512 24.0 / 27.1,
//    fp32 32768 x 160 18.5 / 22.6) nor for bf16 sums alone, which wait for instructions (16384 x 1024 8.3 / 12.4, 32768 x 512
//    9.0 / 13.4), unless every SM has a block (8192 x 2048 out of memory 13.4 / 12.0).  Sums alone of up to 4 MB always
//    (131072 x 8 fp32 12.4 / 10.4).
//  - Single elements, 16 bytes apart in neighbouring lanes: a gradient to store repays its launches for one round of the
//    block's threads (bf16 512 x 1001 12.4 / 10.4, 1024 x 1001 12.4 / 14.0, 8191 x 4095 with the products around it 265 / 399);
//    sums alone for a few (fp32 16384 x 1 6.2 / 6.2, 32768 x 64 behind an odd address 8.0 / 13.1, bf16 8192 x 100 6.2 / 7.2), for
//    eight times as many in wide ranges with a block to every SM (fp32 32768 x 1001 36 / 31, bf16 4096 x 4095 15.5 / 14.4).
inline bool column_cluster_pays(long long rows, long long cols, int size, bool grad, bool aligned) {
  const int v = 16 / size;
  const ColumnPlan p = column_plan(rows, cols, v);
  const long long bytes = rows * cols * size, blocks = p.ranges * p.split, per_block = (bytes + blocks - 1) / blocks;
  const long long narrow = (cols + 2 * v - 1) / (2 * v);  // ranges of 32 bytes
  if (p.ranges > 0x7fffffffLL || (narrow * 8 < column_sms() && bytes > (4 << 20))) return false;
  const bool full = blocks >= column_sms(), wide = p.lanes == 8;
  if (cols % v != 0 || !aligned) {
    const long long at_once = kColumnThreads / p.lanes, rounds = ((rows + p.split - 1) / p.split + at_once - 1) / at_once;
    return rounds <= (grad ? 1 : (size == 4 ? 8 : 2) * (full && wide ? 8 : 1));
  }
  if (per_block <= (96 << 10) || (!grad && bytes <= (4 << 20))) return true;
  if (!grad && size == 2) return full && per_block <= (128 << 10);
  return wide || (p.lanes == 4 && (full || size == 4));
}
template <class Rows>
int launch_colsum(const Rows& m, float* out, long long rows, long long cols, int accumulate, cudaStream_t stream) {
  const ColumnPlan p = column_plan(rows, cols, Rows::kV);
  const dim3 grid(static_cast<unsigned>(p.ranges), static_cast<unsigned>(p.split));
  const long long rpb = (rows + p.split - 1) / p.split;
  const auto kernel = p.lanes == 8   ? colsum_cluster_kernel<Rows, 8>
                      : p.lanes == 4 ? colsum_cluster_kernel<Rows, 4>
                                     : colsum_cluster_kernel<Rows, 2>;
  return launch_column_cluster(kernel, grid, stream, m, out, rows, cols, rpb, accumulate);
}

}  // namespace
}  // namespace fb
