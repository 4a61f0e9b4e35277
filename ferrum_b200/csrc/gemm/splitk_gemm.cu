// bf16 GEMM for outputs of few tiles and a long reduction (sm_100a): weight gradients of small layers over many rows.
// The persistent kernels give such an output to a handful of SMs, each walking the whole reduction alone: 16 x 4096 x
// 4096 took 33 us on 16 SMs where the larger operand streams from HBM in 5.  Here the K splits of a
// tile are one thread-block cluster: every CTA multiplies its share of the k-blocks, the partial tiles meet in
// distributed shared memory in a fixed order, and the epilogue (bias, activation, its derivative, accumulation) runs
// once on the sum.  No workspace, no second launch, no atomics.
//
// What bounds it: one read of the larger operand from HBM.  Two CTAs share an SM with 98 KB of stages each, 29 MB in
// flight over the chip.  Operands in L2, against the persistent kernels: 16 x 4096 x 4096 22.3 -> 9.3 us, 512 x 512 x
// 4096 25.9 -> 11.9, 1024 x 1024 x 8192 (weight gradient) 47.4 -> 25.4.
//
// The tensor core multiplies 128 rows at a time whatever their use.  With up to 64 rows of A (a head of few classes) the
// operands change places: 128 rows of B against a tile of 16, 32 or 64 rows of A, so almost nothing is padding and B is
// read once; the tile is turned round on its way to shared memory.
//
// Few rows of A on the 128-row side need no more than MMAs of 64 rows, whose reads of shared memory (what paces so narrow an
// MMA) are half as many: 33 instead of 44 cycles each.  A programmatic dependent is let in when the last MMA has been issued,
// not before: its CTAs, though they only wait, slowed the issue here from 54 to 81 cycles per MMA (16 x 4096 x 4096 in a
// row 15.6 us, 12.6 so, 12.2 with 64 rows; eight layers of 4096 with their normalisations at 16 rows 183 -> 157).
// Then the producer set the pace, a copy of 2 or 4 KB for every operand of a k-block: where K is whole k-blocks, one copy
// brings a stage of an operand (3-D maps): 12.2 -> 11.0, the eight layers 157 -> 147.
//
// 192 threads: warp 0 TMA producer, warp 1 MMA issue, warps 2 - 5 read the accumulator; all of them write the output.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../common/ptx.cuh"
#include "../common/status.h"
#include "../common/tmem_share.h"
#include "../include/ferrum_kernels.h"
#include "epilogue.cuh"

namespace fb {
namespace {

namespace cg = cooperative_groups;

constexpr int kRowsP = 128;   // rows of the operand on the 128-row side of the MMA
constexpr int kBK = 64;       // one 128-byte swizzle row of bf16
constexpr int kThreads = 192;
constexpr int kMaxStages = 32;
constexpr int kSmemAlone = 200 * 1024, kSmemShared = 98 * 1024;  // stages of a CTA that has its SM alone, or half of it
constexpr int kChunk = 64 * 128;  // 64 rows of 128 bytes: one block of an MN-major operand

template <int BN>
struct Cfg {
  static constexpr int kP = kRowsP * 128;  // what the MMA reads; Args::p_bytes of it are loaded
  static constexpr int kQ = (BN < 64 ? 64 : BN) * 128;  // an MN-major operand arrives in blocks of 64 columns
  static constexpr int kTile = (kRowsP + 4) * (BN + 4) * 4;
  static constexpr int kTmemCols = BN < 32 ? 32 : BN;
};

struct Args {
  void* out;
  void* out2;  // act'(z), stored like out
  const float* bias;
  int M, N;
  long long ldc;
  int p_mn, q_mn;  // operand stored with its rows contiguous
  int out_bf16, act, beta;
  int kb_total, kb_per_split, tiles_p;
  int stages, block_bytes, body_bytes, p_bytes;  // block: a k-block of both operands
  int mma_rows;  // 128, or 64 where P has no more
  int prefetch;  // bring this CTA's rows of B into L2 before the kernel ahead has completed
  int32_t* status;
  unsigned long long timeout_ns;
};

__device__ __forceinline__ float act_of(float x, int act) {
  switch (act) {
    case FB_ACT_RELU: return act_value<FB_ACT_RELU>(x);
    case FB_ACT_GELU: return act_value<FB_ACT_GELU>(x);
    case FB_ACT_SILU: return act_value<FB_ACT_SILU>(x);
    case FB_ACT_TANH: return act_value<FB_ACT_TANH>(x);
    case FB_ACT_SIGMOID: return act_value<FB_ACT_SIGMOID>(x);
    default: return x;
  }
}

__device__ __forceinline__ void store_bf16(void* out, long long at, const float (&f)[4], int count, bool vec) {
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out) + at;
  const __nv_bfloat162 lo = __floats2bfloat162_rn(f[0], f[1]), hi = __floats2bfloat162_rn(f[2], f[3]);
  if (vec) {
    *reinterpret_cast<uint2*>(o) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  } else {
    const __nv_bfloat16 h[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < count) o[j] = h[j];
  }
}

// kSwap: P = B (rows are output columns), Q = A.  kGroup: k-blocks per stage.  One thread issues the MMAs, and a wait,
// a commit and a loop around every four of them take it longer (400 cycles) than the MMAs of a narrow tile (160).
// kBoxes: the kGroup k-blocks of an operand arrive in one copy (3-D maps: 64 of K, rows, k-blocks), those of P, then those of Q;
// else a copy or more for each.  Not a switch at run time: its test in the loops of the two issuing threads cost 35 ns per
// k-block (64 x 64 x 65536 39.0 us, without it 34.5).
template <int BN, bool kSwap, int kGroup, bool kBoxes>
__global__ void __launch_bounds__(kThreads, 2)
gemm_splitk_kernel(const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_q,
                   const __grid_constant__ Args p) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + p.body_bytes);
  uint64_t* empty_bar = full_bar + kMaxStages;
  uint64_t* acc_full = empty_bar + kMaxStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  cg::cluster_group cluster = cg::this_cluster();
  const int splits = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int tile_id = static_cast<int>(blockIdx.x) / splits;
  const int p0 = (tile_id % p.tiles_p) * kRowsP, q0 = (tile_id / p.tiles_p) * BN;
  const int kb_lo = min(p.kb_total, rank * p.kb_per_split), kb_hi = min(p.kb_total, kb_lo + p.kb_per_split);

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(&full_bar[s], 1);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    ptx::mbar_init(acc_full, 1);
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&map_p);
    ptx::prefetch_tensormap(&map_q);
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, C::kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (p.prefetch && warp == 2 && ptx::elect_one()) {
    if constexpr (kBoxes) {
      for (int kb = kb_lo; kb < kb_hi; kb += kGroup) ptx::tma_prefetch_3d(kSwap ? &map_p : &map_q, 0, kSwap ? p0 : q0, kb);
    } else {
      for (int kb = kb_lo; kb < kb_hi; ++kb) ptx::tma_prefetch_2d(kSwap ? &map_p : &map_q, kb * kBK, kSwap ? p0 : q0);
    }
  }
  ptx::grid_wait();

  if (warp == 0) {
    if (ptx::elect_one()) {
      int issued = 0, s = 0;
      uint32_t phase = 1;
      bool ok = true;
      for (int kb = kb_lo; kb < kb_hi; kb += kGroup, ++issued) {
        if (!ptx::mbar_wait(&empty_bar[s], phase, abort_flag, p.timeout_ns)) {
          report_status(p.status, kStatusGemmTimeout, 23, blockIdx.x, kb);
          ok = false;
          break;
        }
        if constexpr (kBoxes) {  // k-blocks behind the last one arrive as zeros
          uint8_t* stage = smem + s * kGroup * p.block_bytes;
          ptx::mbar_arrive_expect_tx(&full_bar[s], kGroup * p.block_bytes);
          ptx::tma_load_3d(stage, &map_p, &full_bar[s], 0, p0, kb);
          ptx::tma_load_3d(stage + kGroup * p.p_bytes, &map_q, &full_bar[s], 0, q0, kb);
        }
        const int blocks = kBoxes ? 0 : min(kGroup, kb_hi - kb);
        if constexpr (!kBoxes) ptx::mbar_arrive_expect_tx(&full_bar[s], blocks * p.block_bytes);
        for (int i = 0; i < blocks; ++i) {
          uint8_t* sp = smem + (s * kGroup + i) * p.block_bytes;
          uint8_t* sq = sp + p.p_bytes;
          const int k0 = (kb + i) * kBK;
          if (p.p_mn) {
#pragma unroll
            for (int c = 0; c < kRowsP / 64; ++c) ptx::tma_load_2d(sp + c * kChunk, &map_p, &full_bar[s], p0 + c * 64, k0);
          } else {
            ptx::tma_load_2d(sp, &map_p, &full_bar[s], k0, p0);
          }
          if (p.q_mn) {
#pragma unroll
            for (int c = 0; c < C::kQ / kChunk; ++c)
              ptx::tma_load_2d(sq + c * kChunk, &map_q, &full_bar[s], q0 + c * 64, k0);
          } else {
            ptx::tma_load_2d(sq, &map_q, &full_bar[s], k0, q0);
          }
        }
        if (++s == p.stages) {
          s = 0;
          phase ^= 1;
        }
      }
      if (!ok) {  // no copy may still be writing shared memory when the CTA goes on: wait (bounded) for those in flight
        for (int i = 0; i < p.stages && i < issued; ++i) {
          const int last = (issued - 1 - i) / p.stages;
          const uint64_t t0 = ptx::globaltimer();
          while (!ptx::mbar_try_wait(&full_bar[i], last & 1))
            if (ptx::globaltimer() - t0 > p.timeout_ns) break;
        }
      }
    }
  } else if (warp == 1) {
    if (kb_hi > kb_lo && ptx::elect_one()) {
      const uint32_t idesc = ptx::make_idesc(1u, p.mma_rows, BN, p.p_mn, p.q_mn);
      const uint32_t p_lbo = p.p_mn ? kChunk : 16, q_lbo = p.q_mn ? kChunk : 16;
      const uint32_t p_step = p.p_mn ? 16 * 128 : 32, q_step = p.q_mn ? 16 * 128 : 32;
      const uint64_t p_first = ptx::make_smem_desc_sw128(ptx::smem_u32(smem), p_lbo, 1024);
      const uint64_t q_first = ptx::make_smem_desc_sw128(ptx::smem_u32(smem) + (kBoxes ? kGroup : 1) * p.p_bytes, q_lbo, 1024);
      int s = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb_lo; kb < kb_hi; kb += kGroup) {
        if (!ptx::mbar_wait(&full_bar[s], phase, abort_flag, p.timeout_ns)) {
          report_status(p.status, kStatusGemmTimeout, 24, blockIdx.x, kb);
          ok = false;
          break;
        }
        ptx::tc_fence_after();
        const auto block = [&](int i) {
          const int at = (s * kGroup + (kBoxes ? 0 : i)) * p.block_bytes;
          const uint64_t dp = ptx::desc_advance(p_first, at + (kBoxes ? i * p.p_bytes : 0));
          const uint64_t dq = ptx::desc_advance(q_first, at + (kBoxes ? i * (p.block_bytes - p.p_bytes) : 0));
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)
            ptx::umma_f16(tmem, ptx::desc_advance(dp, k * p_step), ptx::desc_advance(dq, k * q_step), idesc,
                          (kb - kb_lo) | i | k ? 1u : 0u);
        };
        if (kGroup == 1 || kb + kGroup <= kb_hi) {
#pragma unroll
          for (int i = 0; i < kGroup; ++i) block(i);
        } else {
          for (int i = 0; i < kb_hi - kb; ++i) block(i);
        }
        ptx::umma_commit(&empty_bar[s]);
        if (++s == p.stages) {
          s = 0;
          phase ^= 1;
        }
      }
      if (ok) ptx::umma_commit(acc_full);
      ptx::grid_launch_dependents();
    }
  }

  // ------------------------------------------------------------------ the accumulator as an [m][n] tile of fp32
  constexpr int kRows = kSwap ? BN : kRowsP, kCols = kSwap ? kRowsP : BN, kPitch = kCols + 4;
  float* tile = reinterpret_cast<float*>(smem);
  if (warp >= 2) {
    bool have = kb_hi > kb_lo;
    if (have) {  // every MMA has completed, hence every copy too: the stages are free
      const bool ready = ptx::mbar_wait(acc_full, 0, abort_flag, p.timeout_ns);
      if (!__all_sync(0xffffffffu, ready)) {
        if (lane == 0) report_status(p.status, kStatusGemmTimeout, 25, blockIdx.x, warp);
        have = false;
      }
      ptx::tc_fence_after();
    }
    // rows of the accumulator in tensor memory: 32 to a quarter of the lanes, or 16 (the lower half) of 64
    const int row = (warp & 3) * (p.mma_rows / 4) + lane;
    const bool held = lane < p.mma_rows / 4;
    const uint32_t taddr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll
    for (int j = 0; j < BN / 16; ++j) {
      uint32_t r[16];
      if (have) {
        ptx::tmem_ld_32x32b_x16(taddr + j * 16, r);
        ptx::tmem_wait_ld();
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = 0;
      }
      if constexpr (kSwap) {
#pragma unroll
        for (int i = 0; i < 16; ++i) tile[(j * 16 + i) * kPitch + row] = __uint_as_float(r[i]);
      } else if (held) {
        float4* t4 = reinterpret_cast<float4*>(tile + row * kPitch + j * 16);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          t4[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]),
                              __uint_as_float(r[4 * i + 3]));
      }
    }
  }
  cluster.sync();

  // ------------------------------------------------------------------ add the splits, epilogue
  const int m0 = kSwap ? q0 : p0, n0 = kSwap ? p0 : q0;
  const int esz = p.out_bf16 ? 2 : 4;
  const bool vec = p.N % 4 == 0 && p.ldc % 4 == 0 && reinterpret_cast<uintptr_t>(p.out) % (4 * esz) == 0 &&
                   reinterpret_cast<uintptr_t>(p.out2) % 8 == 0;
  constexpr int kVec = kCols / 4, kAll = kRows * kVec;
  const int share = (kAll + splits - 1) / splits;
  for (int i = rank * share + threadIdx.x; i < min(kAll, (rank + 1) * share); i += kThreads) {
    const int row = i / kVec, c = (i % kVec) * 4;
    const int m = m0 + row, n = n0 + c;
    if (m >= p.M || n >= p.N) continue;
    float f[4] = {0.f, 0.f, 0.f, 0.f};
    for (int r = 0; r < splits; ++r) {
      const float4 t = *reinterpret_cast<const float4*>(cluster.map_shared_rank(tile, r) + row * kPitch + c);
      f[0] += t.x; f[1] += t.y; f[2] += t.z; f[3] += t.w;
    }
    const int count = min(4, p.N - n);
    if (p.bias != nullptr) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < count) f[j] += __ldg(p.bias + n + j);
    }
    const long long at = m * p.ldc + n;
    if (p.out2 != nullptr) {
      float d[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) act_both(f[j], p.act, f[j], d[j]);
      store_bf16(p.out2, at, d, count, vec);
    } else if (p.act != FB_ACT_NONE) {
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = act_of(f[j], p.act);
    }
    if (p.out_bf16) {
      store_bf16(p.out, at, f, count, vec);
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
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < count) o[j] = p.beta ? o[j] + f[j] : f[j];
    }
  }
  ptx::tc_fence_before();
  cluster.sync();  // no CTA leaves while another one still reads its tile
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, C::kTmemCols);
  }
}

// ------------------------------------------------------------ host side
typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                             const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encoder() {
  // The encoder wants a current context; an autograd worker entering its first backward has none yet.
  static thread_local bool bound = false;
  if (!bound) {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaSetDevice(dev);
    bound = true;
  }
  static const EncodeFn fn = [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      sym = nullptr;
    return reinterpret_cast<EncodeFn>(sym);
  }();
  return fn;
}

// `rows` x K operand: boxes of 64 k x `box_rows` rows (K-major) or 64 rows x 64 k (MN-major), 128-byte swizzle.
bool make_map(CUtensorMap* map, const void* ptr, int rows, int K, long long ld, bool mn, int box_rows) {
  const EncodeFn enc = encoder();
  if (enc == nullptr || (reinterpret_cast<uintptr_t>(ptr) & 15) != 0 || ld % 8 != 0) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(mn ? rows : K), static_cast<cuuint64_t>(mn ? K : rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(mn ? 64 : box_rows)}, estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The same of a K-major operand whose K is whole k-blocks, `blocks` of them in a box.
bool make_map_blocks(CUtensorMap* map, const void* ptr, int rows, int K, long long ld, int box_rows, int blocks) {
  const EncodeFn enc = encoder();
  if (enc == nullptr || (reinterpret_cast<uintptr_t>(ptr) & 15) != 0 || ld % 8 != 0) return false;
  const cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(K / 64)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld) * 2, 128};
  const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_rows), static_cast<cuuint32_t>(blocks)}, estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
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

int tiles_of(int rows, int per) { return (rows + per - 1) / per; }

// Tile: 16, 32, 64 = rows of A against 128 rows of B; 128 + 64 or 128 + 128 = 128 rows of A against 64 or 128 of B,
// the wide one where the narrow one leaves no room for four splits (1024 x 1024 x 4096: 18 against 20 us).
int choose_tile(int M, int N) {
  if (M <= 64) return M <= 16 ? 16 : M <= 32 ? 32 : 64;
  return static_cast<long long>(tiles_of(M, kRowsP)) * tiles_of(N, 64) * 4 <= 2 * sm_count() ? 192 : 256;
}

long long tile_count(int M, int N, int tile) {
  return tile <= 64 ? static_cast<long long>(tiles_of(N, kRowsP)) * tiles_of(M, tile)
                    : static_cast<long long>(tiles_of(M, kRowsP)) * tiles_of(N, tile - 128);
}

// As many splits as the two CTAs per SM have room for, each with at least two k-blocks to overlap.
int choose_splits(long long tiles, int kb_total) {
  int splits = 1;
  while (splits < 8 && tiles * splits * 2 <= 2 * sm_count() && splits * 4 <= kb_total) splits *= 2;
  return splits;
}

template <int BN, bool kSwap, int kGroup, bool kBoxes = false>
int launch(const CUtensorMap& mp, const CUtensorMap& mq, Args& g, int rows_p, int rows_q, int box_p, bool split,
           cudaStream_t st) {
  using C = Cfg<BN>;
  constexpr int kExtra = 1024 + 768;  // alignment, barriers
  static const cudaError_t configured = cudaFuncSetAttribute(
      gemm_splitk_kernel<BN, kSwap, kGroup, kBoxes>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemAlone + kExtra);
  if (configured != cudaSuccess) return static_cast<int>(configured);
  g.tiles_p = tiles_of(rows_p, kRowsP);
  const long long tiles = static_cast<long long>(g.tiles_p) * tiles_of(rows_q, BN);
  if (tiles > (1 << 27)) return -1;
  const int splits = split ? choose_splits(tiles, g.kb_total) : 1;
  g.kb_per_split = (g.kb_total + splits - 1) / splits;
  g.p_bytes = box_p * 128;
  g.block_bytes = g.p_bytes + (g.q_mn ? C::kQ : BN * 128);
  g.mma_rows = kSwap || rows_p > 64 ? kRowsP : 64;
  const int tail = g.mma_rows * 128 > g.p_bytes ? g.mma_rows * 128 - g.p_bytes : 0;  // the MMA's reads of rows that were not loaded stay inside the allocation
  // Half an SM for narrow tiles, too: the next one's CTAs start beside this one's.
  const int room = ((split && tiles * splits <= sm_count() ? kSmemAlone : kSmemShared) - tail) / g.block_bytes;
  g.prefetch = !split && (kSwap ? !g.p_mn : !g.q_mn);
  const int need = (g.kb_per_split + kGroup - 1) / kGroup;
  g.stages = room / kGroup < kMaxStages ? room / kGroup : kMaxStages;
  if (g.stages > need) g.stages = need;
  g.body_bytes = (g.stages * kGroup * g.block_bytes + tail + 1023) / 1024 * 1024;
  if (g.body_bytes < C::kTile) g.body_bytes = (C::kTile + 1023) / 1024 * 1024;
  if (splits > 1 && g.body_bytes < kClusterLeastSmem) g.body_bytes = kClusterLeastSmem;  // never, with stages of 18 KB and more
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles * splits));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = g.body_bytes + kExtra;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = splits;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = split ? 1 : 2;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, gemm_splitk_kernel<BN, kSwap, kGroup, kBoxes>, mp, mq, g));
}

}  // namespace
}  // namespace fb

// Where this kernel is the faster one by enough to repay another order of summation.  The persistent kernels take, for any
// output that fits one wave, 4.6 us and 4.3 ns per unit of K on single CTAs and 5.2 us and 2.9 ns on pairs (512 x 512: K 1024
// 8.1, K 4096 16.8 us); this one has 5 to 6 us of launch, cluster and epilogue and then divides K by the splits.  K 256: 6
// against 5.7 us; K 1024: 7 against 9 at best; K 2048: 8 against 13.5 us with eight splits (8 x 4096), 10.8 against 14 with
// four (96 x 4096).  Two splits of a very long reduction stay here although the pairs have caught up since (512 x 4096 x
// 8192 was 43 against 49 us): half the chain of truncating additions, half the error.
extern "C" int fb_gemm_bf16_splitk_use(int M, int N, int K) {
  using namespace fb;
  if (M <= 0 || N <= 0 || K < 2048) return 0;
  const int kb = (K + kBK - 1) / kBK;
  const int splits = choose_splits(tile_count(M, N, choose_tile(M, N)), kb);
  return splits >= 4 || (kb >= 128 && splits >= 2);
}

namespace fb {
namespace {

int run(bool split, const void* a, const void* b, void* out, void* out2, const float* bias, int M, int N, int K,
        long long lda, long long ldb, long long ldc, int a_mn_major, int b_mn_major, int out_bf16, int act, int beta,
        int tile, int32_t* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return -1;
  if ((out2 != nullptr && !out_bf16) || (out_bf16 && beta)) return -1;
  if (tile == 0) tile = choose_tile(M, N);
  if (tile != 16 && tile != 32 && tile != 64 && tile != 160 && tile != 192 && tile != 256) return -1;
  const bool swap = tile <= 64;
  const int bn = swap ? tile : tile - 128;
  // Few rows of A on the 128-row side: only they are loaded (what else the MMA reads there goes into rows of the
  // accumulator that nobody stores).
  const int box_p = swap || a_mn_major || M > 64 ? kRowsP : M <= 16 ? 16 : M <= 32 ? 32 : 64;
  // Stages of four k-blocks while 98 KB hold three of them (boxes of 16 rows of A).
  const bool four = !split && !(swap ? a_mn_major : b_mn_major) && box_p <= 16;
  const int group = tile == 160 ? (four ? 4 : 2) : tile == 192 && four ? 2 : 1;
  CUtensorMap ma, mb;
  Args g;
  const bool boxes = group > 1 && !a_mn_major && !b_mn_major && K % kBK == 0;
  if (boxes) {
    if (!make_map_blocks(&ma, a, M, K, lda, box_p, group) || !make_map_blocks(&mb, b, N, K, ldb, bn, group)) return -2;
  } else if (!make_map(&ma, a, M, K, lda, a_mn_major != 0, swap ? bn : box_p) ||
      !make_map(&mb, b, N, K, ldb, b_mn_major != 0, swap ? kRowsP : bn))
    return -2;
  g.out = out;
  g.out2 = out2;
  g.bias = bias;
  g.M = M;
  g.N = N;
  g.ldc = ldc;
  g.p_mn = swap ? b_mn_major : a_mn_major;
  g.q_mn = swap ? a_mn_major : b_mn_major;
  g.out_bf16 = out_bf16;
  g.act = act;
  g.beta = beta;
  g.kb_total = (K + kBK - 1) / kBK;
  g.status = status;
  g.timeout_ns = 2000000000ull;
  switch (tile) {
    case 16: return launch<16, true, 1>(mb, ma, g, N, M, box_p, split, stream);
    case 32: return launch<32, true, 1>(mb, ma, g, N, M, box_p, split, stream);
    case 64: return launch<64, true, 1>(mb, ma, g, N, M, box_p, split, stream);
    case 160:
      if (boxes)
        return four ? launch<32, false, 4, true>(ma, mb, g, M, N, box_p, split, stream)
                    : launch<32, false, 2, true>(ma, mb, g, M, N, box_p, split, stream);
      return four ? launch<32, false, 4>(ma, mb, g, M, N, box_p, split, stream)
                  : launch<32, false, 2>(ma, mb, g, M, N, box_p, split, stream);
    case 192:
      if (boxes) return launch<64, false, 2, true>(ma, mb, g, M, N, box_p, split, stream);
      return four ? launch<64, false, 2>(ma, mb, g, M, N, box_p, split, stream)
                  : launch<64, false, 1>(ma, mb, g, M, N, box_p, split, stream);
    default: return launch<128, false, 1>(ma, mb, g, M, N, box_p, split, stream);
  }
}

}  // namespace
}  // namespace fb

extern "C" int fb_gemm_bf16_splitk(const void* a, const void* b, void* out, void* out2, const float* bias, int M, int N,
                                   int K, long long lda, long long ldb, long long ldc, int a_mn_major, int b_mn_major,
                                   int out_bf16, int act, int beta, int tile, int32_t* status, cudaStream_t stream) {
  return fb::run(true, a, b, out, out2, bias, M, N, K, lda, ldb, ldc, a_mn_major, b_mn_major, out_bf16, act, beta, tile,
                 status, stream);
}

// Results of up to 64 rows whose sums may not change with the shape (forward passes, input gradients): narrow tiles and
// one chain of MMAs over the whole reduction, the persistent kernels' bits.  Operands from HBM, persistent kernels /
// tiles of 128 columns of B (operands exchanged) / of 32, us: 16 x 4096 x 4096 29.7 / 22.7 / 17.1, 16 x 1024 x 4096
// 29.0 / 20.0 / 13.8, 16 x 4096 x 1024 12.4 / 9.6 / 7.9, 64 x 1000 x 1024 12.8 / 11.0 / 8.4; 16 x 10000 x 1024, more
// tiles of 32 than SMs: 13.0 / 11.3 / 14.9, with 64 columns 10.1.  16 x 128 x 512 was 12.3 on the persistent kernels and
// 14.3 here, 128 x 512 x 512 18.4 on both.  Since then (copies of a whole stage, MMAs of 64 rows, dependents let in after the
// last MMA), operands in L2: 16 x 4096 x 4096 15.6 -> 10.9, 16 x 4096 x 1024 7.2 -> 5.7, 64 x 1000 x 1024 7.3 -> 6.8.
extern "C" int fb_gemm_bf16_narrow_use(int M, int N, int K) {
  return M > 0 && M <= 64 && N >= 512 && N <= fb::kRowsP * fb::sm_count() && K >= 512;
}

extern "C" int fb_gemm_bf16_narrow(const void* a, const void* b, void* out, void* out2, const float* bias, int M, int N,
                                   int K, long long lda, long long ldb, long long ldc, int a_mn_major, int b_mn_major,
                                   int out_bf16, int act, int beta, int tile, int32_t* status, cudaStream_t stream) {
  // The narrowest tile that one wave holds: a CTA's loop is bound by its own copies and MMAs, and the rows of A that every
  // CTA reads again are few.  (An MN-major B arrives in blocks of 64 columns.)
  if (tile == 0 && !b_mn_major && fb::tiles_of(N, 32) <= fb::sm_count()) tile = 160;
  if (tile == 0 && !b_mn_major && fb::tiles_of(N, 64) <= fb::sm_count()) tile = 192;
  if (tile == 0) tile = M <= 32 ? fb::choose_tile(M, N) : 192;
  return fb::run(false, a, b, out, out2, bias, M, N, K, lda, ldb, ldc, a_mn_major, b_mn_major, out_bf16, act, beta, tile,
                 status, stream);
}
