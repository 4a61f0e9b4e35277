// fp32 GEMM on the tensor cores without giving up fp32 precision (sm_100a).
//
// Every fp32 operand element is split into three bf16 numbers a = a0 + a1 + a2, each the value that was left rounded
// to nearest (8 + 8 + 8 significant bits), and six of the nine products are accumulated in fp32 by tcgen05.mma: a0 b0,
// a0 b1, a1 b0, a1 b1, a0 b2, a2 b0.  The three that are left out are below 2^-26 of |a b|, less than the rounding of one
// fp32 multiply-add.  bf16 ends at 2^-133, fp32 at 2^-149: operands are multiplied by 2^16 before the split and sums by
// 2^-32 after it (both exact), so that a = a0 + a1 + a2 holds for every finite value down to the last subnormal.  The tensor core truncates where it adds (2048 x 2048 x 4096 of
// normal numbers summed there alone: relative error 2.8e-5), so each k-block of 64 gets a fresh accumulator and the
// k-blocks are added in registers, rounded to nearest: 1.7e-7, against 1.1e-6 of a chain of fp32 multiply-adds.
//
// What bounds it: the split, about eight instructions per operand element in sixteen warps and most of them in the integer
// pipe (2700 cycles per k-block of a 128 x 128 tile, where the six bf16 MMAs per fp32 product take 1536: 271 TFLOP/s at the
// measured bf16 rate).  It happens on the way from global memory (registers) to the tensor core, so any element strides are
// accepted, nothing is staged in global memory and no second launch is needed.  The planes of A go to tensor memory, those of B
// to shared memory (three bf16 planes, 128-byte swizzle): with both in shared memory the MMAs' reads and the split's stores
// came to 2304 cycles of its bandwidth and a k-block to 3000.  A thread's elements of A are the ones that it may write to
// tensor memory, in pieces that are still read 64 bytes a row (load_a).  B with contiguous rows keeps them in shared memory
// (kVecRow): vector loads instead of eight single ones per piece, 1024^3 20.6 -> 18.9 us.
//
// One CTA per 128 x BN output tile and K split.  The splits of a tile are one thread-block cluster: the partial tiles
// meet through distributed shared memory in a fixed order, so small outputs fill the chip without a workspace.
//
// Infinities, NaNs and values that would round to infinity (from 2^112) do not survive the split (inf - inf, 0 * inf) and
// always end in a result that is not finite, and so do sums above 2^96; such a result is computed again with fp32
// multiply-adds when the tile is written.
//
// bf16 operands whose rows a TMA map cannot describe (a pitch that is no multiple of 16 bytes, an odd base) take the
// same kernel with one plane and one product: no padded copies, no fp32 copies.  Rows at any 2-byte address are read
// with aligned 16-byte loads and shifted into place; the loads and the shifts bound it, not the MMAs.  Against fp32
// copies on the multiply-add kernel: 777 x 1001 x 1001 17 instead of 148 us, 8191 x 4095 x 4095 1.3 (both K-major) to
// 1.8 ms (both row-major) instead of 12.4; relative error 9e-8 instead of 2.5e-7 at K = 1001.  Large operands are laid out
// again and take the aligned kernels: with a bf16 result any, with an fp32 result those whose reduction is a multiple of 8
// (native/core.cpp, repack_repays and copies_repay).
//
// The issue of a k-block's MMAs takes as long as the MMAs themselves (the queue is short), so it has a warp of its own;
// a loader warp that issued them held up the next stage (5200 instead of 2300 cycles per k-block).  The first loads are
// on their way before barriers and tensor memory are set up, tiles without splits meet without a cluster barrier, and the
// partial sums are asked for several at a time.  us before all this and now: 1024 x 1024 x 64 8.8 / 6.2, 1024^3 21.1 / 19.2, 2048^3
// 114 / 104, 591 x 1536 x 384 15.4 / 13.0, 128 x 256 x 784 8.8 / 7.6, 1 x 256 x 784 7.6 / 6.6.  Large products run into the
// power limit.  8192 x 4096 x 4096, forward, input gradient and weight gradient: 1549 / 1482 by itself; in rows of sixty at the
// limit, the two sides taking turns, 1820 / 1756, 1983 / 1726 and 1905 / 1940 (whoever comes first on a cool chip is 5 % faster);
// a training step of three layers of 4096 over 8192 rows 14.7 / 13.9 ms.  Seventeen warps leave 96 registers: with A's rows
// contiguous (weight gradients) tiles of 128 spill 36 - 40 bytes, 20 - 28 before.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cfloat>
#include <cstdint>

#include "../common/ptx.cuh"
#include "../common/status.h"
#include "../common/tmem_share.h"
#include "../include/ferrum_kernels.h"

namespace fb {
namespace {

namespace cg = cooperative_groups;

constexpr float kUp = 65536.f, kDown = 1.f / (kUp * kUp);  // of an operand before the split, of a sum after it

constexpr int kBM = 128;
constexpr int kBlock = 64 * 128;  // 64 rows (k) of 128 bytes: a block of an operand with its rows contiguous
constexpr int kLoaders = 512;
constexpr int kThreads = kLoaders + 32;  // 16 warps load, split, add up and write; one issues the MMAs

// The element type of the operands: fp32 in three bf16 planes, or bf16 in one.
template <typename T>
struct El;
template <>
struct El<float> {
  struct Piece {
    float v[8];
  };
  static constexpr int kPlanes = 3, kProducts = 6;
};
template <>
struct El<__nv_bfloat16> {
  struct Piece {
    uint32_t w[8];  // as loaded: words, the two words that cover a piece at an odd address, or single elements
    uint32_t off;   // byte offset of the piece in w
  };
  static constexpr int kPlanes = 1, kProducts = 1;
};

template <typename T, int BN>
struct Cfg {
  static constexpr int kBK = 64;                   // elements of K per stage
  static constexpr int kRow = kBK * 2;             // bytes of a row of a bf16 plane = its swizzle width
  static constexpr int kPieces = kBK / 8;          // 8-element pieces per row
  static constexpr int kPlaneA = kBM * kRow, kPlaneB = BN * kRow;
  static constexpr bool kATmem = El<T>::kPlanes > 1;   // the planes of A lie in tensor memory
  static constexpr int kStage = El<T>::kPlanes * kPlaneB + (kATmem ? 0 : El<T>::kPlanes * kPlaneA);
  static constexpr int kStages = kATmem && BN == 128 ? 2 : 4;
  static constexpr int kPlaneCols = kBK / 2;           // columns of tensor memory of a plane of A
  static constexpr int kPitch = BN + 4;   // floats per row of the tile in shared memory: conflict-free 16-byte rows
  static constexpr int kTile = kBM * kPitch * 4;
  static constexpr int kBody = kStages * kStage > kTile ? kStages * kStage : kTile;
  static constexpr int kSmem = kBody + 1024 + 256;
  // With splits: all of tensor memory is held over a cluster barrier (common/tmem_share.h).  The registers alone (96 x 544)
  // kept other such CTAs off the SM until here.
  static constexpr int kSmemSplit = kATmem && kSmem < kClusterAloneSmem ? kClusterAloneSmem : kSmem;
  static constexpr int kTmemCols = kATmem ? 512 : 2 * BN;  // two accumulators, then the stages of A
  static_assert(kSmem >= kClusterLeastSmem, "tensor memory is held over a cluster barrier");
  static_assert(kTmemCols < 512 || kSmemSplit + kClusterLeastSmem + 2 * kCtaSmem > kSmSmem, "no room for another one's columns");
  static constexpr int kPerThread = (kATmem ? BN : kBM + BN) * kPieces / kLoaders;  // pieces of a stage per thread
  static constexpr int kAcc = kBM * BN / kLoaders;                    // accumulators per thread: a quarter of a tile row
  // 16-byte chunk of a row, as the 128- / 64-byte swizzle of the matrix descriptors places it
  __device__ static uint32_t at(int row, int kc) {
    return row * kRow + ((kc ^ (kRow == 128 ? row & 7 : (row >> 1) & 3)) << 4);
  }
  __device__ static uint64_t desc(uint32_t addr) {
    return ptx::make_smem_desc_sw128(addr, 16, 8 * kRow, kRow == 128 ? 2 : 4);
  }
};

struct Operand {
  const void* p;
  long long s_row, s_k, s_bo, s_bi;  // element strides; slices of the batch (outer, inner)
  int rows;
  uintptr_t end;                     // address past the last element
};

// How an operand lies in memory: K contiguous with 16-byte aligned rows (two vector loads per piece), K contiguous
// with any alignment, anything else (lanes follow the rows), or (fp32, B) rows contiguous with 16-byte aligned steps of K: a
// piece is then eight rows at one k, and the tile in shared memory has its rows contiguous, too.
enum Layout { kVecK = 0, kScalarK = 1, kRowFast = 2, kVecRow = 3 };

struct Args {
  Operand a, b;
  void* out;
  const float* bias;
  long long ldc, sc_bo, sc_bi;
  int M, N, K;
  int act, beta, out_bf16;
  float alpha;
  int batch_inner;
  int kb_total, kb_per_split;
  int32_t* status;
  unsigned long long timeout_ns;
};

__device__ __forceinline__ float act_f(float x, int act) {
  switch (act) {
    case FB_ACT_RELU: return fmaxf(x, 0.f);
    case FB_ACT_GELU: {
      const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
      return 0.5f * x * (1.f + tanhf(u));
    }
    case FB_ACT_SILU: return x / (1.f + expf(-x));
    case FB_ACT_TANH: return tanhf(x);
    case FB_ACT_SIGMOID: return 1.f / (1.f + expf(-x));
    default: return x;
  }
}

template <typename T>
__device__ __noinline__ float dot_again(const T* a, long long sa, const T* b, long long sb, int K) {
  float s = 0.f;
  for (int k = 0; k < K; ++k) s = fmaf(a[k * sa], b[k * sb], s);
  return s;
}

// Where piece `c` of an operand tile (row, 8 consecutive k) lies: neighbouring lanes follow the contiguous direction.
template <int ROWS, int L, int PIECES>
__device__ __forceinline__ void piece(int c, int& row, int& kc) {
  if (L == kRowFast) {
    row = c % ROWS;
    kc = c / ROWS;
  } else if (L == kVecRow) {  // eight rows from `row` at k = kc
    row = c % (ROWS / 8) * 8;
    kc = c / (ROWS / 8);
  } else {
    row = c / PIECES;
    kc = c % PIECES;
  }
}

// Rows past the edge read the last row (their products are dropped with the tile's edge), so whole k-blocks load
// without a condition and stay in flight until they are split; only the last k-block of a ragged K is guarded.
template <int ROWS, int L, int PIECES>
__device__ __forceinline__ void load_piece(const Operand& o, const float* base, int row0, int k0, int K, int c,
                                           El<float>::Piece& out) {
  float(&v)[8] = out.v;
  int row, kc;
  piece<ROWS, L, PIECES>(c, row, kc);
  if constexpr (L == kVecRow) {
    // Octets outside the tile's edge are kept off the single loads, which their warp would else take after the vector loads, in
    // the form that costs the fewest registers: in 128 rows they read the last octet again (for columns that nobody stores), in
    // 64 they go by quads.  us with single loads for all of them / so: weight gradients 16 x 32 over 100000 rows 290 / 269, 128 x
    // 72 over 20000 65.6 / 61.6, 1000 x 1000 over 2048 41.0 / 39.0, its input gradient 36.9 / 32.9.
    const int k = k0 + kc, r = ROWS > 64 && o.rows % 8 == 0 ? min(row0 + row, o.rows - 8) : row0 + row;
    const float* p = base + k * o.s_k + r;
    if constexpr (ROWS > 64) {
      if (k < K && r + 8 <= o.rows) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(p)), y = __ldg(reinterpret_cast<const float4*>(p) + 1);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] = 0.f;
          if (k < K && r + j < o.rows) v[j] = __ldg(p + j);
        }
      }
    } else {
      const int left = k < K ? o.rows - r : 0;
#pragma unroll
      for (int q = 0; q < 8; q += 4) {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (left >= q + 4) {
          x = __ldg(reinterpret_cast<const float4*>(p + q));
        } else if (left > q) {
          x.x = __ldg(p + q);
          if (left > q + 1) x.y = __ldg(p + q + 1);
          if (left > q + 2) x.z = __ldg(p + q + 2);
        }
        v[q] = x.x; v[q + 1] = x.y; v[q + 2] = x.z; v[q + 3] = x.w;
      }
    }
    return;
  }
  const int r = min(row0 + row, o.rows - 1), k = k0 + kc * 8;
  if (k0 + PIECES * 8 <= K) {
    if constexpr (L == kVecK) {
      const float* p = base + r * o.s_row + k;
      const float4 x = __ldg(reinterpret_cast<const float4*>(p)), y = __ldg(reinterpret_cast<const float4*>(p) + 1);
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
      v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    } else if constexpr (L == kScalarK) {
      const float* p = base + r * o.s_row + k;
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __ldg(p + j);
    } else {
      const float* p = base + r * o.s_row + k * o.s_k;
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __ldg(p + j * o.s_k);
    }
  } else {
    const float* p = base + r * o.s_row;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = 0.f;
      if (k + j < K) v[j] = __ldg(p + (k + j) * o.s_k);
    }
  }
}

__device__ __forceinline__ uint32_t u16_at(const __nv_bfloat16* p) {
  return __ldg(reinterpret_cast<const unsigned short*>(p));
}

// The same for bf16.  A row at an odd address: the two aligned 16-byte words that cover the piece, if both lie inside
// the operand; element by element at the operand's first and last bytes.  Words are kept as they arrive and put
// together when they are stored, so that nothing waits for a load here.
template <int ROWS, int L, int PIECES>
__device__ __forceinline__ void load_piece(const Operand& o, const __nv_bfloat16* base, int row0, int k0, int K, int c,
                                           El<__nv_bfloat16>::Piece& v) {
  int row, kc;
  piece<ROWS, L, PIECES>(c, row, kc);
  const int r = min(row0 + row, o.rows - 1), k = k0 + kc * 8;
  const __nv_bfloat16* p = base + r * o.s_row + k * o.s_k;
  auto quad = [&](int i, uintptr_t at) {
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(at));
    v.w[i] = x.x; v.w[i + 1] = x.y; v.w[i + 2] = x.z; v.w[i + 3] = x.w;
  };
  const bool whole = k0 + PIECES * 8 <= K;
  if (L == kVecK && whole) {
    quad(0, reinterpret_cast<uintptr_t>(p));
  } else if (L == kRowFast) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v.w[j] = 0;
      if (whole || k + j < K) v.w[j] = u16_at(p + j * o.s_k);
    }
  } else {
    const uintptr_t at = reinterpret_cast<uintptr_t>(p), lo = at & ~uintptr_t(15);
    if (L == kScalarK && whole && lo >= reinterpret_cast<uintptr_t>(o.p) && lo + 32 <= o.end) {
      quad(0, lo);
      quad(4, lo + 16);
      v.off = static_cast<uint32_t>(at & 15);
    } else {
      uint32_t e[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        e[j] = 0;
        if (whole || k + j < K) e[j] = u16_at(p + j);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) v.w[j] = e[2 * j] | e[2 * j + 1] << 16;
      v.off = 0;
    }
  }
}

__device__ __forceinline__ float2 sub2(float2 x, float2 y) {  // x - y with one packed instruction: y * -1 is exact
  float2 r;
  asm("{\n.reg .b64 a, b, c, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %6};\n"
      "fma.rn.f32x2 d, b, c, a;\nmov.b64 {%0, %1}, d;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y), "f"(-1.f));
  return r;
}
__device__ __forceinline__ float2 add2(float2 x, float2 y) {
  float2 r;
  asm("{\n.reg .b64 a, b, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nadd.rn.f32x2 d, a, b;\nmov.b64 {%0, %1}, d;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y));
  return r;
}
__device__ __forceinline__ float2 scale2(float2 x, float s) {
  float2 r;
  asm("{\n.reg .b64 a, b, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %4};\nmul.rn.f32x2 d, a, b;\nmov.b64 {%0, %1}, d;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x.x), "f"(x.y), "f"(s));
  return r;
}
__device__ __forceinline__ uint32_t bf16_pair(float2 x) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x.x, x.y);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 wide_pair(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}

// Two values scaled and split: a word of each plane.
__device__ __forceinline__ void split_pair(float x0, float x1, uint32_t& w0, uint32_t& w1, uint32_t& w2) {
  const float2 x = scale2(make_float2(x0, x1), kUp);
  w0 = bf16_pair(x);
  const float2 r = sub2(x, wide_pair(w0));
  w1 = bf16_pair(r);
  w2 = bf16_pair(sub2(r, wide_pair(w1)));
}

// Splits a thread's share of A (load_a) into the planes at `at`: the lanes of its warp, the columns of its slice of K.
template <int L, int PLANE>
__device__ __forceinline__ void store_a(uint32_t at, const float (&v)[16]) {
  uint32_t w0[8], w1[8], w2[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) split_pair(v[2 * j], v[2 * j + 1], w0[j], w1[j], w2[j]);
  if constexpr (L == kRowFast) {
    ptx::tmem_st_32x32b_x8(at, w0);
    ptx::tmem_st_32x32b_x8(at + PLANE, w1);
    ptx::tmem_st_32x32b_x8(at + 2 * PLANE, w2);
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t to = at + (static_cast<uint32_t>(16 * h) << 16);
      ptx::tmem_st_16x256b(to, w0[4 * h], w0[4 * h + 1], w0[4 * h + 2], w0[4 * h + 3]);
      ptx::tmem_st_16x256b(to + PLANE, w1[4 * h], w1[4 * h + 1], w1[4 * h + 2], w1[4 * h + 3]);
      ptx::tmem_st_16x256b(to + 2 * PLANE, w2[4 * h], w2[4 * h + 1], w2[4 * h + 2], w2[4 * h + 3]);
    }
  }
}

// Splits eight values and stores them into the three planes.
template <int L>
__device__ __forceinline__ void store_piece(uint32_t at, uint32_t plane_bytes, const El<float>::Piece& in) {
  const float(&v)[8] = in.v;
  uint32_t w0[4], w1[4], w2[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) split_pair(v[2 * j], v[2 * j + 1], w0[j], w1[j], w2[j]);
  ptx::st_shared_v4(at, w0[0], w0[1], w0[2], w0[3]);
  ptx::st_shared_v4(at + plane_bytes, w1[0], w1[1], w1[2], w1[3]);
  ptx::st_shared_v4(at + 2 * plane_bytes, w2[0], w2[1], w2[2], w2[3]);
}

template <int L>
__device__ __forceinline__ void store_piece(uint32_t at, uint32_t, const El<__nv_bfloat16>::Piece& v) {
  if constexpr (L == kVecK) {
    ptx::st_shared_v4(at, v.w[0], v.w[1], v.w[2], v.w[3]);
  } else if constexpr (L == kRowFast) {
    ptx::st_shared_v4(at, v.w[0] | v.w[1] << 16, v.w[2] | v.w[3] << 16, v.w[4] | v.w[5] << 16, v.w[6] | v.w[7] << 16);
  } else {
    uint32_t t[6], s[5];
#pragma unroll
    for (int i = 0; i < 6; ++i) t[i] = v.off & 8 ? v.w[i + 2] : v.w[i];
#pragma unroll
    for (int i = 0; i < 5; ++i) s[i] = v.off & 4 ? t[i + 1] : t[i];
    const uint32_t sh = (v.off & 2) * 8;
    ptx::st_shared_v4(at, __funnelshift_r(s[0], s[1], sh), __funnelshift_r(s[1], s[2], sh),
                      __funnelshift_r(s[2], s[3], sh), __funnelshift_r(s[3], s[4], sh));
  }
}

// A thread's share of a k-block of A on its way to tensor memory: 16 elements of 32 rows x 16 of K (the rows are the lanes
// that its warp may write, the slice of K is its warp's).  K contiguous: four rows, four elements each, as tmem_st_16x256b
// places them, so that four lanes read 64 bytes of a row; rows contiguous: one row each (tmem_st_32x32b_x8).
template <int L>
__device__ __forceinline__ void load_a(const Operand& o, const float* base, int row0, int k0, int K, float (&v)[16]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kw = k0 + (warp >> 2) * 16;
  row0 += (warp & 3) * 32;
  const bool whole = k0 + 64 <= K;
  if constexpr (L == kRowFast) {
    const float* p = base + min(row0 + lane, o.rows - 1) * o.s_row + kw * o.s_k;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      v[j] = 0.f;
      if (whole || kw + j < K) v[j] = __ldg(p + j * o.s_k);
    }
  } else {
    const int k = kw + (lane & 3) * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float* p = base + min(row0 + i * 8 + (lane >> 2), o.rows - 1) * o.s_row + k;
      if (L == kVecK && whole) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(p));
        v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[4 * i + j] = 0.f;
          if (whole || k + j < K) v[4 * i + j] = __ldg(p + j);
        }
      }
    }
  }
}

template <typename T, int BN, int LA, int LB>
__global__ void __launch_bounds__(kThreads, 1) gemm_split_kernel(const __grid_constant__ Args p) {
  using C = Cfg<T, BN>;
  constexpr int kPlanes = El<T>::kPlanes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + C::kBody);
  uint64_t* empty_bar = full_bar + C::kStages;
  uint64_t* acc_full = empty_bar + C::kStages;   // accumulator buffer complete
  uint64_t* acc_empty = acc_full + 2;            // accumulator buffer read out
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  cg::cluster_group cluster = cg::this_cluster();
  const int splits = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());

  const int n0 = static_cast<int>(blockIdx.x / splits) * BN, m0 = static_cast<int>(blockIdx.y) * kBM;
  const int bo = static_cast<int>(blockIdx.z) / p.batch_inner, bi = static_cast<int>(blockIdx.z) % p.batch_inner;
  const T* a = static_cast<const T*>(p.a.p) + bo * p.a.s_bo + bi * p.a.s_bi;
  const T* b = static_cast<const T*>(p.b.p) + bo * p.b.s_bo + bi * p.b.s_bi;
  const long long out_at = bo * p.sc_bo + bi * p.sc_bi;

  const int kb_lo = min(p.kb_total, rank * p.kb_per_split), kb_hi = min(p.kb_total, kb_lo + p.kb_per_split);
  const int nkb = kb_hi - kb_lo;

  // The first k-block's loads are on their way before barriers and tensor memory are set up.
  constexpr int kPA = C::kATmem ? 0 : kBM * C::kPieces / kLoaders;  // pieces of A per thread; the rest are B's
  typename El<T>::Piece v[C::kPerThread];
  float va[C::kATmem ? 16 : 1];
  auto fetch_a = [&](int kb) {
    if constexpr (C::kATmem) load_a<LA>(p.a, a, m0, kb * C::kBK, p.K, va);
  };
  auto fetch = [&](int i, int kb) {
    const int k0 = kb * C::kBK;
    if (i < kPA)
      load_piece<kBM, LA, C::kPieces>(p.a, a, m0, k0, p.K, i * kLoaders + threadIdx.x, v[i]);
    else
      load_piece<BN, LB, C::kPieces>(p.b, b, n0, k0, p.K, (i - kPA) * kLoaders + threadIdx.x, v[i]);
  };
  if (warp < kLoaders / 32 && nkb > 0) {
    fetch_a(kb_lo);
#pragma unroll
    for (int i = 0; i < C::kPerThread; ++i) fetch(i, kb_lo);
  }
  if (threadIdx.x == kLoaders) {
    *abort_flag = 0;
    for (int s = 0; s < C::kStages; ++s) {
      ptx::mbar_init(&full_bar[s], kLoaders / 32);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&acc_full[i], 1);
      ptx::mbar_init(&acc_empty[i], kLoaders / 32);
    }
    ptx::fence_mbar_init();
  }
  if (warp == kLoaders / 32) {
    __syncwarp();
    ptx::tmem_alloc(tmem_slot, C::kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  float acc[C::kAcc];
  if (warp < kLoaders / 32) {
    // -------------------------------------------------------- load, split, add up
#pragma unroll
    for (int i = 0; i < C::kAcc; ++i) acc[i] = 0.f;
    const uint32_t taddr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + (warp >> 2) * C::kAcc;
    int blocks_read = 0;
    bool ok = true;
    auto read_block = [&]() {  // adds a finished k-block's accumulator to the registers
      const int buf = blocks_read & 1;
      const bool ready = ptx::mbar_wait(&acc_full[buf], (blocks_read >> 1) & 1, abort_flag, p.timeout_ns);
      if (!__all_sync(0xffffffffu, ready)) {
        ok = false;
        return;
      }
      ptx::tc_fence_after();
#pragma unroll
      for (int j = 0; j < C::kAcc / 16; ++j) {
        uint32_t r[16];
        ptx::tmem_ld_32x32b_x16(taddr + buf * BN + j * 16, r);
        ptx::tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const float2 s = add2(make_float2(acc[j * 16 + i], acc[j * 16 + i + 1]),
                                make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])));
          acc[j * 16 + i] = s.x;
          acc[j * 16 + i + 1] = s.y;
        }
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&acc_empty[buf]);
      ++blocks_read;
    };
    for (int kb = 0; kb < nkb && ok; ++kb) {
      const int s = kb % C::kStages;
      const bool free_slot = ptx::mbar_wait(&empty_bar[s], ((kb / C::kStages) & 1) ^ 1, abort_flag, p.timeout_ns);
      if (!__all_sync(0xffffffffu, free_slot)) {
        ok = false;
        break;
      }
      const uint32_t sa = ptx::smem_u32(smem + s * C::kStage), sb = C::kATmem ? sa : sa + kPlanes * C::kPlaneA;
      const bool more = kb + 1 < nkb;
      if constexpr (C::kATmem) {
        ptx::tc_fence_after();
        store_a<LA, C::kPlaneCols>(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + 2 * BN +
                                       s * kPlanes * C::kPlaneCols + (warp >> 2) * 8, va);
        if (more) fetch_a(kb_lo + kb + 1);
      }
#pragma unroll
      for (int i = 0; i < C::kPerThread; ++i) {
        int row, kc;
        if (i < kPA) {
          piece<kBM, LA, C::kPieces>(i * kLoaders + threadIdx.x, row, kc);
          store_piece<LA>(sa + C::at(row, kc), C::kPlaneA, v[i]);
        } else {
          piece<BN, LB, C::kPieces>((i - kPA) * kLoaders + threadIdx.x, row, kc);
          // rows contiguous: blocks of 64 rows, 128 bytes per k
          const int at = LB == kVecRow ? (row >> 6) * kBlock + C::at(kc, (row >> 3) & 7) : C::at(row, kc);
          store_piece<LB>(sb + at, C::kPlaneB, v[i]);
        }
        if (more) fetch(i, kb_lo + kb + 1);
      }
      ptx::fence_proxy_async_smem();
      if constexpr (C::kATmem) {
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&full_bar[s]);
      if (kb > 0) read_block();  // the k-block before: added up while the MMAs of this one run
    }
    if (ok && nkb > 0) read_block();
    if (!ok) {
      if (lane == 0) report_status(p.status, kStatusGemmTimeout, 21, blockIdx.x, warp);
    }
  } else if (ptx::elect_one()) {
    // ---------------------------------------------------------------- MMA issue
    const uint32_t idesc = ptx::make_idesc(1u, kBM, BN, 0, LB == kVecRow ? 1 : 0);
    const uint64_t first = LB == kVecRow ? ptx::make_smem_desc_sw128(ptx::smem_u32(smem), kBlock, 1024)
                                         : C::desc(ptx::smem_u32(smem));
    constexpr int kStepB = LB == kVecRow ? 16 * 128 : 32;  // 16 of K
    for (int kb = 0; kb < nkb; ++kb) {
      const int s = kb % C::kStages, buf = kb & 1;
      if (!ptx::mbar_wait(&acc_empty[buf], ((kb >> 1) & 1) ^ 1, abort_flag, p.timeout_ns) ||
          !ptx::mbar_wait(&full_bar[s], (kb / C::kStages) & 1, abort_flag, p.timeout_ns)) {
        report_status(p.status, kStatusGemmTimeout, 22, blockIdx.x, kb);
        break;
      }
      ptx::tc_fence_after();
      const uint64_t da = ptx::desc_advance(first, s * C::kStage);
      const uint64_t db = C::kATmem ? da : ptx::desc_advance(da, kPlanes * C::kPlaneA);
      const uint32_t ta = tmem + 2 * BN + s * kPlanes * C::kPlaneCols;
      const uint32_t d = tmem + buf * BN;
      constexpr int ia[6] = {2, 0, 1, 1, 0, 0}, ib[6] = {0, 2, 1, 0, 1, 0};  // small products first
      constexpr int kFirst = 6 - El<T>::kProducts;
#pragma unroll
      for (int q = kFirst; q < 6; ++q) {
#pragma unroll
        for (int k = 0; k < C::kBK / 16; ++k) {
          const uint64_t dbk = ptx::desc_advance(db, ib[q] * C::kPlaneB + k * kStepB);
          const uint32_t sum = (q != kFirst || k != 0) ? 1u : 0u;
          if constexpr (C::kATmem)
            ptx::umma_f16_ta(d, ta + ia[q] * C::kPlaneCols + k * 8, dbk, idesc, sum);
          else
            ptx::umma_f16(d, ptx::desc_advance(da, ia[q] * C::kPlaneA + k * 32), dbk, idesc, sum);
        }
      }
      ptx::umma_commit(&empty_bar[s]);
      ptx::umma_commit(&acc_full[buf]);
    }
  }

  // ------------------------------------------------------------------ partial tiles meet
  // Every MMA of this CTA has completed (the loaders waited for the last one), so its stages hold the tile.
  float* tile = reinterpret_cast<float*>(smem);
  const int rows_per = kBM / splits;  // what this CTA adds up and writes
  if (warp < kLoaders / 32) {
    float4* t4 = reinterpret_cast<float4*>(tile + ((warp & 3) * 32 + lane) * C::kPitch + (warp >> 2) * C::kAcc);
#pragma unroll
    for (int i = 0; i < C::kAcc / 4; ++i)
      t4[i] = make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
  }
  ptx::tc_fence_before();
  if (splits > 1) cluster.sync();
  else __syncthreads();
  if (warp == kLoaders / 32) {
    ptx::tc_fence_after();
    __syncwarp();
    ptx::tmem_dealloc(tmem, C::kTmemCols);
  }
  const int esz = p.out_bf16 ? 2 : 4;
  const bool vec = p.N % 4 == 0 && p.ldc % 4 == 0 && out_at % 4 == 0 && reinterpret_cast<uintptr_t>(p.out) % (4 * esz) == 0;
  constexpr int kVec = BN / 4, kRowStep = kLoaders / kVec;
  const int c = static_cast<int>(threadIdx.x) % kVec * 4, n = n0 + c;
  const int row0 = rank * rows_per, rows = warp < kLoaders / 32 && n < p.N ? min(rows_per, p.M - m0 - row0) : 0;
  float bias[4] = {0.f, 0.f, 0.f, 0.f};
  if (p.bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < p.N) bias[j] = __ldg(p.bias + n + j);
  }
  // Added up in the order of the splits, with several reads (of the other CTAs' tiles) on their way at a time: two rows of up
  // to two splits, or one row of them all.
  const int step = splits > 2 ? kRowStep : 2 * kRowStep;
  for (int l0 = threadIdx.x / kVec; l0 < rows; l0 += step) {
    const bool two = splits <= 2 && l0 + kRowStep < rows;
    const int at0 = (row0 + l0) * C::kPitch + c;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f), next = sum;
    if (splits > 2) {
      float4 part[8];
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < splits) part[r] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(tile, r) + at0);
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < splits) {
          sum.x += part[r].x; sum.y += part[r].y; sum.z += part[r].z; sum.w += part[r].w;
        }
    } else {
#pragma unroll 2
      for (int r = 0; r < splits; ++r) {
        const float* from = cluster.map_shared_rank(tile, r) + at0;
        const float4 x = *reinterpret_cast<const float4*>(from);
        const float4 y = *reinterpret_cast<const float4*>(from + (two ? kRowStep * C::kPitch : 0));
        sum.x += x.x; sum.y += x.y; sum.z += x.z; sum.w += x.w;
        next.x += y.x; next.y += y.y; next.z += y.z; next.w += y.w;
      }
    }
#pragma unroll 1
    for (int u = 0; u <= static_cast<int>(two); ++u) {
      const int m = m0 + row0 + l0 + u * kRowStep;
      float f[4] = {sum.x, sum.y, sum.z, sum.w};
      sum = next;
      if constexpr (kPlanes > 1) {
        bool finite = true;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          finite &= fabsf(f[j]) <= FLT_MAX;
          f[j] *= kDown;
        }
        // not finite: an operand that does not survive the split, or a result that is not finite in fp32 either
        if (!finite) {
#pragma unroll 1
          for (int j = 0; j < 4; ++j) {  // the four values change places instead of being indexed
            float y = f[0];
            if (!(fabsf(y) <= FLT_MAX) && n + j < p.N)
              y = dot_again(a + m * p.a.s_row, p.a.s_k, b + (n + j) * p.b.s_row, p.b.s_k, p.K);
            f[0] = f[1]; f[1] = f[2]; f[2] = f[3]; f[3] = y;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        f[j] *= p.alpha;
        if (p.bias != nullptr) f[j] += bias[j];
      }
      if (p.act != FB_ACT_NONE) {
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {  // one copy of the code, as above
          const float y = act_f(f[0], p.act);
          f[0] = f[1]; f[1] = f[2]; f[2] = f[3]; f[3] = y;
        }
      }
      const long long at = out_at + m * p.ldc + n;
      if (p.out_bf16) {
        __nv_bfloat16* o = static_cast<__nv_bfloat16*>(p.out) + at;
        if (vec) {
          *reinterpret_cast<uint2*>(o) = make_uint2(bf16_pair(make_float2(f[0], f[1])), bf16_pair(make_float2(f[2], f[3])));
        } else {
          for (int j = 0; j < 4 && n + j < p.N; ++j) o[j] = __float2bfloat16_rn(f[j]);
        }
        continue;
      }
      float* o = static_cast<float*>(p.out) + at;
      if (vec) {
        float4 x = make_float4(f[0], f[1], f[2], f[3]);
        if (p.beta) {
          const float4 old = *reinterpret_cast<float4*>(o);
          x.x += old.x; x.y += old.y; x.z += old.z; x.w += old.w;
        }
        *reinterpret_cast<float4*>(o) = x;
      } else {
        for (int j = 0; j < 4 && n + j < p.N; ++j) o[j] = p.beta ? o[j] + f[j] : f[j];
      }
    }
  }
  if (splits > 1) cluster.sync();  // no CTA leaves while another one still reads its tile
}

int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  }
  return n;
}

// Clusters of `size` CTAs that are on the chip at once: fewer than SMs / size, a cluster lies within one part of the chip.
template <typename T, int BN>
int resident_clusters(int size) {
  static std::atomic<int> known[9];
  int n = known[size].load(std::memory_order_relaxed);
  if (n == 0) {
    const auto kernel = gemm_split_kernel<T, BN, kVecK, kVecK>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(size));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = Cfg<T, BN>::kSmemSplit;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = size;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<T, BN>::kSmemSplit) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = sm_count() / size;
    }
    known[size].store(n, std::memory_order_relaxed);
  }
  return n;
}

template <typename T, int BN, int LA, int LB>
int launch_one(const Args& args, int batch, int splits, cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel<T, BN, LA, LB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               Cfg<T, BN>::kSmemSplit);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((args.N + BN - 1) / BN * splits), static_cast<unsigned>((args.M + kBM - 1) / kBM),
                     static_cast<unsigned>(batch));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = splits > 1 ? Cfg<T, BN>::kSmemSplit : Cfg<T, BN>::kSmem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = splits;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, gemm_split_kernel<T, BN, LA, LB>, args));
}

template <typename T, int BN, int LA>
int launch_b(int lb, const Args& args, int batch, int splits, cudaStream_t st) {
  if (lb == kVecK) return launch_one<T, BN, LA, kVecK>(args, batch, splits, st);
  if (lb == kScalarK) return launch_one<T, BN, LA, kScalarK>(args, batch, splits, st);
  if constexpr (El<T>::kPlanes > 1) {
    if (lb == kVecRow) return launch_one<T, BN, LA, kVecRow>(args, batch, splits, st);
  }
  return launch_one<T, BN, LA, kRowFast>(args, batch, splits, st);
}
template <typename T, int BN>
int launch(int la, int lb, const Args& args, int batch, int splits, cudaStream_t st) {
  if (la == kVecK) return launch_b<T, BN, kVecK>(lb, args, batch, splits, st);
  if (la == kScalarK) return launch_b<T, BN, kScalarK>(lb, args, batch, splits, st);
  return launch_b<T, BN, kRowFast>(lb, args, batch, splits, st);
}

template <typename T>
int layout_of(const Operand& o) {
  constexpr int kUnit = 16 / sizeof(T);
  if (o.s_k != 1) return kRowFast;
  return reinterpret_cast<uintptr_t>(o.p) % 16 == 0 && o.s_row % kUnit == 0 && o.s_bo % kUnit == 0 && o.s_bi % kUnit == 0
             ? kVecK
             : kScalarK;
}

// Strides as the callers give them: a (rows M), b (rows N); K, batch and output strides.
template <typename T>
int gemm_split(const T* a, const T* b, void* out, int out_bf16, const float* bias, int M, int N, int K, long long sam,
               long long sak, long long sbn, long long sbk, long long ldc, int act, int beta, float alpha,
               int batch_outer, int batch_inner, long long sa_outer, long long sa_inner, long long sb_outer,
               long long sb_inner, long long sc_outer, long long sc_inner, int32_t* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch_outer <= 0 || batch_inner <= 0) return 0;
  const long long batch = static_cast<long long>(batch_outer) * batch_inner;
  if (K < 0 || batch > 65535 || (M + kBM - 1) / kBM > 65535) return -1;
  auto operand = [&](const T* p, int rows, long long s_row, long long s_k, long long s_bo, long long s_bi) {
    const long long last = (rows - 1) * s_row + (K > 0 ? K - 1 : 0) * s_k + (batch_outer - 1) * s_bo + (batch_inner - 1) * s_bi;
    return Operand{p, s_row, s_k, s_bo, s_bi, rows, reinterpret_cast<uintptr_t>(p + last + 1)};
  };
  Args g;
  g.a = operand(a, M, sam, sak, sa_outer, sa_inner);
  g.b = operand(b, N, sbn, sbk, sb_outer, sb_inner);
  g.out = out;
  g.out_bf16 = out_bf16;
  g.bias = bias;
  g.ldc = ldc;
  g.sc_bo = sc_outer;
  g.sc_bi = sc_inner;
  g.M = M;
  g.N = N;
  g.K = K;
  g.act = act;
  g.beta = beta;
  g.alpha = alpha;
  g.batch_inner = batch_inner;
  g.status = status;
  g.timeout_ns = 2000000000ull;
  // Tile width and K splits: the wide tile where it alone fills the chip, else the narrow one; then as many splits
  // as there are idle SMs, each with at least one k-block, but no more than leave all clusters on the chip at once (16 of
  // eight CTAs do not fit: 1024 x 128 x 2048 took two turns, 22 us, and takes 16.7 with
  // four; 128 x 1024 x 1024 16.4 and 9.8).
  const long long tm = (M + kBM - 1) / kBM;
  const long long wide = tm * ((N + 127) / 128) * batch, narrow = tm * ((N + 63) / 64) * batch;
  constexpr int kBK = Cfg<T, 128>::kBK;
  const bool use_wide = N > 64 && wide * 8 > sm_count() && wide * (K + 127) / 128 >= sm_count();
  const long long tiles = use_wide ? wide : narrow;
  g.kb_total = (K + kBK - 1) / kBK;
  int splits = 1;
  const auto fits = [&](int n) { return tiles <= (use_wide ? resident_clusters<T, 128>(n) : resident_clusters<T, 64>(n)); };
  while (splits < 8 && tiles * splits * 2 <= sm_count() && splits * 2 <= g.kb_total && fits(splits * 2)) splits *= 2;
  g.kb_per_split = (g.kb_total + splits - 1) / splits;
  const int la = layout_of<T>(g.a);
  int lb = layout_of<T>(g.b);
  if (El<T>::kPlanes > 1 && lb == kRowFast && g.b.s_row == 1 && reinterpret_cast<uintptr_t>(g.b.p) % 16 == 0 &&
      g.b.s_k % 4 == 0 && g.b.s_bo % 4 == 0 && g.b.s_bi % 4 == 0)
    lb = kVecRow;
  return use_wide ? launch<T, 128>(la, lb, g, static_cast<int>(batch), splits, stream)
                  : launch<T, 64>(la, lb, g, static_cast<int>(batch), splits, stream);
}

}  // namespace
}  // namespace fb

using namespace fb;

extern "C" int fb_gemm_f32_tensor(const float* a, const float* b, float* out, const float* bias, int M, int N, int K,
                                  long long sam, long long sak, long long sbn, long long sbk, long long ldc, int act,
                                  int beta, float alpha, int batch_outer, int batch_inner, long long sa_outer,
                                  long long sa_inner, long long sb_outer, long long sb_inner, long long sc_outer,
                                  long long sc_inner, int32_t* status, cudaStream_t stream) {
  return gemm_split<float>(a, b, out, 0, bias, M, N, K, sam, sak, sbn, sbk, ldc, act, beta, alpha, batch_outer,
                           batch_inner, sa_outer, sa_inner, sb_outer, sb_inner, sc_outer, sc_inner, status, stream);
}

extern "C" int fb_gemm_bf16_any(const void* a, const void* b, void* out, const float* bias, int M, int N, int K,
                                long long sam, long long sak, long long sbn, long long sbk, long long ldc, int out_bf16,
                                int act, int beta, int32_t* status, cudaStream_t stream) {
  if (out_bf16 && beta) return -1;
  return gemm_split<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(a), static_cast<const __nv_bfloat16*>(b), out,
                                   out_bf16, bias, M, N, K, sam, sak, sbn, sbk, ldc, act, beta, 1.f, 1, 1, 0, 0, 0, 0, 0,
                                   0, status, stream);
}
