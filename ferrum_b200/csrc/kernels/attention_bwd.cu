// Blockwise attention backward on the tcgen05 tensor cores, head dimension 64, bf16: dQ, dK, dV from Q, K, V, dO,
// the row log-sum-exp the forward kernel saved and delta = rowsum(dO * O).  Nothing of size S x S is read from or
// written to memory: the probabilities are recomputed tile by tile from the scores, as in the forward kernel
// (attention.cu).  The reference keeps the whole [S, S] matrix per head (ferrum-nn/src/transformer.rs:127-220).
//
// Two kernels, both shaped like the forward kernel (same operand layouts, same roles), so that neither needs an
// atomic or a cross-CTA reduction:
//
// Roles of a CTA: warp 0 TMA producer, warp 1 MMA issuer, then groups of four warps for the elementwise work (two
// tensor-memory reads, an exponential and half a dozen multiply-adds per score).  The stationary tile has 128 rows, the other
// side is walked 64 at a time: a tile's scores and dP take 128 columns of tensor memory, one group's, and the products of one
// tile run beside the elementwise work of the others.  A group waits for its products longer than they take, so there are as
// many groups as tensor memory holds beside the accumulators: three for a head dimension of 64, two for 128.  8 x 16 heads
// of 64, 1024 rows, two and three groups: dQ 99 / 93 us, dK and dV 140 / 120; the sums over the tiles and their order are the same.
//
//   attn_bwd_dq_kernel    a CTA owns 128 query rows and walks the key / value tiles:
//                           S = Q K_j^T, dP = dO V_j^T            (tensor memory, 2 x 64 columns per group)
//                           dS = P * (dP - delta) * scale          (thread = query row; bf16 into shared memory)
//                           dQ += dS K_j                           (accumulates in tensor memory over all tiles)
//   attn_bwd_dkv_kernel   a CTA owns 128 keys and walks the query tiles, everything transposed:
//                           S^T = K Q_i^T, dP^T = V dO_i^T
//                           P^T, dS^T                              (thread = key row; lse / delta of the tile's
//                                                                   queries come through shared memory)
//                           dV += P^T dO_i,  dK += dS^T Q_i        (accumulate in tensor memory)
//
// The scores are computed twice (once per kernel): 7 tile GEMMs per pair of tiles instead of 5, in exchange for
// kernels without atomics whose every MMA operand layout is one the forward kernel already uses.  Causal masks
// skip the tiles on the far side of the diagonal in both kernels.  Every mbarrier wait is bounded.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <utility>

#include "../common/ptx.cuh"
#include "../common/status.h"
#include "../include/ferrum_kernels.h"

namespace fb {
namespace {

constexpr int kT = 128;                     // rows of the stationary tile
constexpr int kW = 64;                      // rows of a tile of the side that is walked
constexpr int kBlk = kT * 128;              // 16 KB: 128 rows of 64 bf16 = one 128-byte-swizzled block
constexpr int kBlkW = kW * 128;             // the same of 64 rows
constexpr int kTmemBwd = 512;               // scores and dP of the groups, 128 columns each; then the accumulators
// D = head dimension (64 or 128).  An operand tile is D / 64 blocks side by side.
template <int D>
struct BwdCfg {
  static constexpr int kNB = D / 64;
  static constexpr int kTile = kNB * kBlk, kTileW = kNB * kBlkW;
  static constexpr int kG = D == 64 ? 3 : 2;       // groups of four softmax warps: as many as tensor memory has room for
  static constexpr int kThreads = 64 + kG * 128;   // TMA warp, MMA warp, groups
  static constexpr int kStages = D == 64 ? 5 : 3;  // a tile's scores are issued kG tiles ahead of its release
  static constexpr int kSmemDq = 2 * kTile + 2 * kStages * kTileW + kG * kBlk + 1024 + 256;  // Q dO | K V | dS
  // K V | Q dO | P^T dS^T | lse, delta
  static constexpr int kSmemDkv = 2 * kTile + 2 * kStages * kTileW + 2 * kG * kBlk + kG * 2 * kW * 4 + 1024 + 256;
};

// One operand tile: D / 64 boxes of 64 columns, `bytes` each.
template <int D>
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int row0, int h, int b,
                                          int bytes) {
#pragma unroll
  for (int nb = 0; nb < D / 64; ++nb) ptx::tma_load_4d(dst + nb * bytes, map, bar, nb * 64, row0, h, b);
}
// Given up: no copy may outlive the CTA (bounded).  `issued` tiles went through the ring.
__device__ __forceinline__ void drain(uint64_t* fixed, uint64_t* full, int issued, int stages, unsigned long long timeout_ns) {
  const uint64_t t0 = ptx::globaltimer();
  while (!ptx::mbar_try_wait(fixed, 0) && ptx::globaltimer() - t0 <= timeout_ns) {
  }
  for (int st = 0; st < stages && st < issued; ++st)
    while (!ptx::mbar_try_wait(&full[st], ((issued - 1 - st) / stages) & 1) && ptx::globaltimer() - t0 <= timeout_ns) {
    }
}
constexpr float kLog2e = 1.4426950408889634f;

struct BwdArgs {
  __nv_bfloat16* dq;   // [B, Sq, H, D]
  __nv_bfloat16* dk;   // [B, Skv, H, D]
  __nv_bfloat16* dv;   // [B, Skv, H, D]
  const float* lse;    // [B, H, Sq] natural log
  const float* delta;  // [B, H, Sq]
  int B, H, Sq, Skv;
  float scale, scale_log2;
  int causal;
  int32_t* status;
  unsigned long long timeout_ns;
};

__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 128 x 64 x D product of two K-major tiles (rows x D): the score shape.
template <int D>
__device__ __forceinline__ void mma_scores(uint32_t tmem, uint32_t a, uint32_t b, uint32_t idesc) {
  const uint64_t da = ptx::make_smem_desc_sw128(a, 16, 1024), db = ptx::make_smem_desc_sw128(b, 16, 1024);
#pragma unroll
  for (int k = 0; k < D / 16; ++k)
    ptx::umma_f16(tmem, ptx::desc_advance(da, (k >> 2) * kBlk + (k & 3) * 32),
                  ptx::desc_advance(db, (k >> 2) * kBlkW + (k & 3) * 32), idesc, k != 0 ? 1u : 0u);
}
// 128 x D x 64 product: A = a 128 x 64 matrix, K-major, B = a 64 x D tile whose D columns are contiguous (MN-major; its
// 64-column blocks lie kBlkW apart): the P V shape of the forward kernel.
__device__ __forceinline__ void mma_pv(uint32_t tmem, uint32_t a, uint32_t b, uint32_t idesc, bool accumulate) {
  const uint64_t da = ptx::make_smem_desc_sw128(a, 16, 1024), db = ptx::make_smem_desc_sw128(b, kBlkW, 1024);
#pragma unroll
  for (int k = 0; k < kW / 16; ++k)
    ptx::umma_f16(tmem, ptx::desc_advance(da, k * 32), ptx::desc_advance(db, k * 2048), idesc,
                  (accumulate || k != 0) ? 1u : 0u);
}

// 16 columns (8 bf16 pairs) of one row of a 128 x 64 matrix, starting at column col (a multiple of 16): two 16-byte chunks
// of the row's 128-byte line, swizzled.
__device__ __forceinline__ void store_cols16(uint8_t* mat, int row, int col, const uint32_t (&w)[8]) {
  uint8_t* line = mat + row * 128;
  const int chunk = col >> 3;
  *reinterpret_cast<uint4*>(line + (((chunk) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
  *reinterpret_cast<uint4*>(line + (((chunk + 1) ^ (row & 7)) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
}
// The 64 columns of a tile in four batches of 16: the tensor-memory loads of batch k + 1 are in flight while batch k is
// computed (tcgen05.wait::ld waits for every load issued before it, so the wait for a batch comes after the arithmetic of
// the previous one).
template <class Batch>
__device__ __forceinline__ void walk_columns(uint32_t t_s, uint32_t t_dp, Batch batch) {
  uint32_t sa[16], pa[16], sb[16], pb[16];
  ptx::tmem_ld_32x32b_x16(t_s, sa);
  ptx::tmem_ld_32x32b_x16(t_dp, pa);
  ptx::tmem_wait_ld();
  ptx::tmem_ld_32x32b_x16(t_s + 16, sb);
  ptx::tmem_ld_32x32b_x16(t_dp + 16, pb);
  batch(0, sa, pa);
  ptx::tmem_wait_ld();
  ptx::tmem_ld_32x32b_x16(t_s + 32, sa);
  ptx::tmem_ld_32x32b_x16(t_dp + 32, pa);
  batch(16, sb, pb);
  ptx::tmem_wait_ld();
  ptx::tmem_ld_32x32b_x16(t_s + 48, sb);
  ptx::tmem_ld_32x32b_x16(t_dp + 48, pb);
  batch(32, sa, pa);
  ptx::tmem_wait_ld();
  batch(48, sb, pb);
}

// Chunks c_lo .. c_hi - 1 (32 columns each) of an accumulator row from tensor memory to bf16 in global memory.  The tensor-memory loads are
// warp-wide (.sync.aligned): EVERY lane of the warp must call this, `valid` only predicates the stores.
__device__ __forceinline__ void store_row_bf16(__nv_bfloat16* dst, uint32_t tmem_row, bool valid, int c_lo,
                                               int c_hi) {
#pragma unroll 1
  for (int c = c_lo; c < c_hi; ++c) {
    uint32_t r[32];
    ptx::tmem_ld_32x32b_x32(tmem_row + c * 32, r);
    ptx::tmem_wait_ld();
    if (!valid) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __nv_bfloat162 pk = __floats2bfloat162_rn(__uint_as_float(r[q * 8 + e * 2]),
                                                        __uint_as_float(r[q * 8 + e * 2 + 1]));
        w[e] = *reinterpret_cast<const uint32_t*>(&pk);
      }
      reinterpret_cast<uint4*>(dst)[c * 4 + q] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// ------------------------------------------------------------------------------------------------ dQ
template <int D>
__global__ void __launch_bounds__(BwdCfg<D>::kThreads, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                   const BwdArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int kTile = BwdCfg<D>::kTile, kTileW = BwdCfg<D>::kTileW, kStages = BwdCfg<D>::kStages, kG = BwdCfg<D>::kG;
  uint8_t* sq = smem;
  uint8_t* sdo = sq + kTile;
  uint8_t* sk = sdo + kTile;              // kStages tiles
  uint8_t* sv = sk + kStages * kTileW;    // kStages tiles
  uint8_t* sds = sv + kStages * kTileW;   // dS of the groups: 128 x 64 bf16 each
  uint64_t* q_full = reinterpret_cast<uint64_t*>(sds + kG * kBlk);
  uint64_t* kv_full = q_full + 1;           // [kStages]
  uint64_t* kv_empty = kv_full + kStages;   // [kStages]
  uint64_t* sp_full = kv_empty + kStages;   // [kG] S and dP of a group's tile are complete
  uint64_t* ds_full = sp_full + kG;         // [kG] dS written (and S, dP read) by the group's four warps
  uint64_t* ds_empty = ds_full + kG;        // [kG] the dQ MMAs have read dS
  uint64_t* dq_full = ds_empty + kG;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(dq_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  // under a causal mask the query tiles with the most keys first
  const int q0 = static_cast<int>(p.causal ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * kT;
  const int h = blockIdx.y % p.H, b = blockIdx.y / p.H;
  const int off = p.Skv - p.Sq;
  const int kv_end = p.causal ? min(p.Skv, q0 + kT + off) : p.Skv;
  const int n_tiles = (kv_end + kW - 1) / kW;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    ptx::mbar_init(q_full, 1);
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(&kv_full[s], 1);
      ptx::mbar_init(&kv_empty[s], 1);
    }
    for (int g = 0; g < kG; ++g) {
      ptx::mbar_init(&sp_full[g], 1);
      ptx::mbar_init(&ds_full[g], 4);
      ptx::mbar_init(&ds_empty[g], 1);
    }
    ptx::mbar_init(dq_full, 1);
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&map_q);
    ptx::prefetch_tensormap(&map_k);
    ptx::prefetch_tensormap(&map_v);
    ptx::prefetch_tensormap(&map_do);
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, kTmemBwd);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t t_dq = tmem_base + kG * 2 * kW;

  if (warp == 0) {
    if (ptx::elect_one()) {
      ptx::mbar_arrive_expect_tx(q_full, 2 * kTile);
      load_tile<D>(sq, &map_q, q_full, q0, h, b, kBlk);
      load_tile<D>(sdo, &map_do, q_full, q0, h, b, kBlk);
      int j = 0;
      for (; j < n_tiles; ++j) {
        const int st = j % kStages;
        if (!ptx::mbar_wait(&kv_empty[st], ((j / kStages) & 1) ^ 1, abort_flag, p.timeout_ns)) {
          report_status(p.status, kStatusGemmTimeout, 61, blockIdx.x, j);
          break;
        }
        ptx::mbar_arrive_expect_tx(&kv_full[st], 2 * kTileW);
        load_tile<D>(sk + st * kTileW, &map_k, &kv_full[st], j * kW, h, b, kBlkW);
        load_tile<D>(sv + st * kTileW, &map_v, &kv_full[st], j * kW, h, b, kBlkW);
      }
      if (j < n_tiles || *abort_flag) drain(q_full, kv_full, j, kStages, p.timeout_ns);
    }
  } else if (warp == 1) {
    if (ptx::elect_one()) {
      const uint32_t idesc_s = ptx::make_idesc(1u, kT, kW, 0, 0);
      const uint32_t idesc_o = ptx::make_idesc(1u, kT, D, 0, 1);
      const uint32_t sq_a = ptx::smem_u32(sq), sdo_a = ptx::smem_u32(sdo), sds_a = ptx::smem_u32(sds);
      const uint32_t sk_a = ptx::smem_u32(sk), sv_a = ptx::smem_u32(sv);
      auto issue_s = [&](int j) {  // S and dP of tile j
        const int st = j % kStages, g = j % kG;
        if (!ptx::mbar_wait(&kv_full[st], (j / kStages) & 1, abort_flag, p.timeout_ns)) {
          report_status(p.status, kStatusGemmTimeout, 63, blockIdx.x, j);
          return false;
        }
        ptx::tc_fence_after();
        mma_scores<D>(tmem_base + g * 2 * kW, sq_a, sk_a + st * kTileW, idesc_s);
        mma_scores<D>(tmem_base + g * 2 * kW + kW, sdo_a, sv_a + st * kTileW, idesc_s);
        ptx::umma_commit(&sp_full[g]);
        return true;
      };
      bool ok = ptx::mbar_wait(q_full, 0, abort_flag, p.timeout_ns);
      if (!ok) report_status(p.status, kStatusGemmTimeout, 62, blockIdx.x, 0);
      for (int j = 0; ok && j < kG && j < n_tiles; ++j) ok = issue_s(j);
      for (int j = 0; ok && j < n_tiles; ++j) {
        const int st = j % kStages, g = j % kG;
        // dS of tile j is written, its S and dP have been read
        if (!ptx::mbar_wait(&ds_full[g], (j / kG) & 1, abort_flag, p.timeout_ns)) {
          report_status(p.status, kStatusGemmTimeout, 64, blockIdx.x, j);
          break;
        }
        ptx::tc_fence_after();
        if (j + kG < n_tiles) {
          ok = issue_s(j + kG);
          if (!ok) break;
        }
        mma_pv(t_dq, sds_a + g * kBlk, sk_a + st * kTileW, idesc_o, j != 0);
        ptx::umma_commit(&kv_empty[st]);
        ptx::umma_commit(&ds_empty[g]);
        if (j + 1 == n_tiles) ptx::umma_commit(dq_full);
      }
    }
  } else {
    const int quarter = warp & 3, g = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;
    const int qrow = q0 + row;
    const uint32_t t_row = (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t t_s = tmem_base + t_row + g * 2 * kW;
    uint8_t* my_ds = sds + g * kBlk;
    const long long stat = (static_cast<long long>(b) * p.H + h) * p.Sq + qrow;
    // a row past the end contributes nothing: +inf makes every probability zero
    const float lse2 = qrow < p.Sq ? p.lse[stat] * kLog2e : INFINITY;
    const float delta = qrow < p.Sq ? p.delta[stat] : 0.f;
    bool ok = true;
    for (int j = g; j < n_tiles; j += kG) {
      const int turn = j / kG;
      // S and dP are there; the dQ MMAs of the group's tile before have read dS
      bool ready = ptx::mbar_wait(&sp_full[g], turn & 1, abort_flag, p.timeout_ns);
      if (ready && turn > 0) ready = ptx::mbar_wait(&ds_empty[g], (turn - 1) & 1, abort_flag, p.timeout_ns);
      if (!__all_sync(0xffffffffu, ready)) {
        if (lane == 0) report_status(p.status, kStatusGemmTimeout, 65, blockIdx.x, j);
        ok = false;
        break;
      }
      ptx::tc_fence_after();
      int valid = min(kW, p.Skv - j * kW);
      if (p.causal) valid = max(0, min(valid, qrow + off + 1 - j * kW));
      {
        const float2 sl2 = make_float2(p.scale_log2, p.scale_log2), nl2 = make_float2(-lse2, -lse2);
        const float2 sc2 = make_float2(p.scale, p.scale), nd2 = make_float2(-delta * p.scale, -delta * p.scale);
        auto batch = [&](int col, const uint32_t (&rs)[16], const uint32_t (&rp)[16]) {
          uint32_t w[8];
          // packed path (two scores per instruction) unless the causal diagonal or the end of the keys cuts a row
          if (__all_sync(0xffffffffu, col + 16 <= valid)) {
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              const float2 e = __ffma2_rn(make_float2(__uint_as_float(rs[i]), __uint_as_float(rs[i + 1])), sl2, nl2);
              const float2 t = __ffma2_rn(make_float2(__uint_as_float(rp[i]), __uint_as_float(rp[i + 1])), sc2, nd2);
              const float2 d = __fmul2_rn(make_float2(ex2f(e.x), ex2f(e.y)), t);
              const __nv_bfloat162 pk = __floats2bfloat162_rn(d.x, d.y);
              w[i >> 1] = *reinterpret_cast<const uint32_t*>(&pk);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              float d0 = 0.f, d1 = 0.f;
              if (col + i < valid)
                d0 = ex2f(fmaf(__uint_as_float(rs[i]), p.scale_log2, -lse2)) * (__uint_as_float(rp[i]) - delta) * p.scale;
              if (col + i + 1 < valid)
                d1 = ex2f(fmaf(__uint_as_float(rs[i + 1]), p.scale_log2, -lse2)) *
                     (__uint_as_float(rp[i + 1]) - delta) * p.scale;
              const __nv_bfloat162 pk = __floats2bfloat162_rn(d0, d1);
              w[i >> 1] = *reinterpret_cast<const uint32_t*>(&pk);
            }
          }
          store_cols16(my_ds, row, col, w);
        };
        walk_columns(t_s, t_s + kW, batch);
      }
      ptx::tc_fence_before();
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&ds_full[g]);
    }
    if (ok && g < 2) {
      const bool done = ptx::mbar_wait(dq_full, 0, abort_flag, p.timeout_ns);
      if (!__all_sync(0xffffffffu, done)) {
        if (lane == 0) report_status(p.status, kStatusGemmTimeout, 67, blockIdx.x, 0);
      } else {
        ptx::tc_fence_after();
        __nv_bfloat16* dst = p.dq + ((static_cast<long long>(b) * p.Sq + qrow) * p.H + h) * D;
        store_row_bf16(dst, t_dq + t_row, qrow < p.Sq, g * (D / 64), (g + 1) * (D / 64));  // a group each half of the columns
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, kTmemBwd);
  }
}

// ------------------------------------------------------------------------------------------------ dK, dV
template <int D>
__global__ void __launch_bounds__(BwdCfg<D>::kThreads, 1)
attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                    const BwdArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int kTile = BwdCfg<D>::kTile, kTileW = BwdCfg<D>::kTileW, kStages = BwdCfg<D>::kStages, kG = BwdCfg<D>::kG;
  uint8_t* sk = smem;
  uint8_t* sv = sk + kTile;
  uint8_t* sq = sv + kTile;               // kStages tiles
  uint8_t* sdo = sq + kStages * kTileW;   // kStages tiles
  uint8_t* spt = sdo + kStages * kTileW;  // P^T of the groups: 128 keys x 64 queries bf16 each
  uint8_t* sdst = spt + kG * kBlk;        // dS^T
  float* s_stat = reinterpret_cast<float*>(sdst + kG * kBlk);  // per group: lse and delta of its tile's 64 queries
  uint64_t* kv_full = reinterpret_cast<uint64_t*>(s_stat + kG * 2 * kW);
  uint64_t* qd_full = kv_full + 1;          // [kStages]
  uint64_t* qd_empty = qd_full + kStages;   // [kStages]
  uint64_t* sp_full = qd_empty + kStages;   // [kG] S^T and dP^T of a group's tile are complete
  uint64_t* pt_full = sp_full + kG;         // [kG] P^T and dS^T written by the group's four warps
  uint64_t* pt_empty = pt_full + kG;        // [kG] the MMAs have read them
  uint64_t* acc_full = pt_empty + kG;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  const int k0 = blockIdx.x * kT;
  const int h = blockIdx.y % p.H, b = blockIdx.y / p.H;
  const int off = p.Skv - p.Sq;
  const int n_qtiles = (p.Sq + kW - 1) / kW;
  // causal: query q sees key k when k <= q + off, so the first query that sees this tile's first key is k0 - off
  const int i_begin = p.causal ? max(0, k0 - off) / kW : 0;
  const int n_iter = max(0, n_qtiles - i_begin);

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    ptx::mbar_init(kv_full, 1);
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(&qd_full[s], 1);
      ptx::mbar_init(&qd_empty[s], 1);
    }
    for (int g = 0; g < kG; ++g) {
      ptx::mbar_init(&sp_full[g], 1);
      ptx::mbar_init(&pt_full[g], 4);
      ptx::mbar_init(&pt_empty[g], 1);
    }
    ptx::mbar_init(acc_full, 1);
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&map_q);
    ptx::prefetch_tensormap(&map_k);
    ptx::prefetch_tensormap(&map_v);
    ptx::prefetch_tensormap(&map_do);
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, kTmemBwd);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t t_dv = tmem_base + kG * 2 * kW, t_dk = t_dv + D;

  if (warp == 0) {
    if (n_iter > 0 && ptx::elect_one()) {
      ptx::mbar_arrive_expect_tx(kv_full, 2 * kTile);
      load_tile<D>(sk, &map_k, kv_full, k0, h, b, kBlk);
      load_tile<D>(sv, &map_v, kv_full, k0, h, b, kBlk);
      int it = 0;
      for (; it < n_iter; ++it) {
        const int st = it % kStages, i = i_begin + it;
        if (!ptx::mbar_wait(&qd_empty[st], ((it / kStages) & 1) ^ 1, abort_flag, p.timeout_ns)) {
          report_status(p.status, kStatusGemmTimeout, 71, blockIdx.x, it);
          break;
        }
        ptx::mbar_arrive_expect_tx(&qd_full[st], 2 * kTileW);
        load_tile<D>(sq + st * kTileW, &map_q, &qd_full[st], i * kW, h, b, kBlkW);
        load_tile<D>(sdo + st * kTileW, &map_do, &qd_full[st], i * kW, h, b, kBlkW);
      }
      if (it < n_iter || *abort_flag) drain(kv_full, qd_full, it, kStages, p.timeout_ns);
    }
  } else if (warp == 1) {
    if (n_iter > 0 && ptx::elect_one()) {
      const uint32_t idesc_s = ptx::make_idesc(1u, kT, kW, 0, 0);
      const uint32_t idesc_o = ptx::make_idesc(1u, kT, D, 0, 1);
      const uint32_t sk_a = ptx::smem_u32(sk), sv_a = ptx::smem_u32(sv), sq_a = ptx::smem_u32(sq), sdo_a = ptx::smem_u32(sdo);
      const uint32_t spt_a = ptx::smem_u32(spt), sdst_a = ptx::smem_u32(sdst);
      auto issue_s = [&](int it) {
        const int st = it % kStages, g = it % kG;
        if (!ptx::mbar_wait(&qd_full[st], (it / kStages) & 1, abort_flag, p.timeout_ns)) {
          report_status(p.status, kStatusGemmTimeout, 73, blockIdx.x, it);
          return false;
        }
        ptx::tc_fence_after();
        mma_scores<D>(tmem_base + g * 2 * kW, sk_a, sq_a + st * kTileW, idesc_s);        // S^T  = K Q_i^T
        mma_scores<D>(tmem_base + g * 2 * kW + kW, sv_a, sdo_a + st * kTileW, idesc_s);  // dP^T = V dO_i^T
        ptx::umma_commit(&sp_full[g]);
        return true;
      };
      bool ok = ptx::mbar_wait(kv_full, 0, abort_flag, p.timeout_ns);
      if (!ok) report_status(p.status, kStatusGemmTimeout, 72, blockIdx.x, 0);
      for (int it = 0; ok && it < kG && it < n_iter; ++it) ok = issue_s(it);
      for (int it = 0; ok && it < n_iter; ++it) {
        const int st = it % kStages, g = it % kG;
        if (!ptx::mbar_wait(&pt_full[g], (it / kG) & 1, abort_flag, p.timeout_ns)) {
          report_status(p.status, kStatusGemmTimeout, 74, blockIdx.x, it);
          break;
        }
        ptx::tc_fence_after();
        if (it + kG < n_iter) {
          ok = issue_s(it + kG);
          if (!ok) break;
        }
        mma_pv(t_dv, spt_a + g * kBlk, sdo_a + st * kTileW, idesc_o, it != 0);   // dV += P^T dO_i
        mma_pv(t_dk, sdst_a + g * kBlk, sq_a + st * kTileW, idesc_o, it != 0);   // dK += dS^T Q_i
        ptx::umma_commit(&qd_empty[st]);
        ptx::umma_commit(&pt_empty[g]);
        if (it + 1 == n_iter) ptx::umma_commit(acc_full);
      }
    }
  } else {
    const int quarter = warp & 3, g = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;   // key row of this thread
    const int krow = k0 + row;
    const uint32_t t_row = (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t t_s = tmem_base + t_row + g * 2 * kW;
    uint8_t *my_pt = spt + g * kBlk, *my_dst = sdst + g * kBlk;
    float* slot = s_stat + g * 2 * kW;
    const long long stat_base = (static_cast<long long>(b) * p.H + h) * p.Sq;
    bool ok = true;
    for (int it = g; it < n_iter; it += kG) {
      const int i = i_begin + it, turn = it / kG;
      float nl[2], nd[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int q = i * kW + x * 32 + lane;
        // negated, so that one fused multiply-add forms the exponent; -inf: a query past the end sees nothing
        nl[x] = q < p.Sq ? -p.lse[stat_base + q] * kLog2e : -INFINITY;
        nd[x] = q < p.Sq ? -p.delta[stat_base + q] * p.scale : 0.f;
      }
      bool ready = ptx::mbar_wait(&sp_full[g], turn & 1, abort_flag, p.timeout_ns);
      if (ready && turn > 0) ready = ptx::mbar_wait(&pt_empty[g], (turn - 1) & 1, abort_flag, p.timeout_ns);
      if (!__all_sync(0xffffffffu, ready)) {
        if (lane == 0) report_status(p.status, kStatusGemmTimeout, 75, blockIdx.x, it);
        ok = false;
        break;
      }
      ptx::tc_fence_after();
      // All four warps write the same values.  The scores of this tile were issued after every one of them was done with
      // the tile before, so nobody reads the slot any more.
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        slot[x * 32 + lane] = nl[x];
        slot[kW + x * 32 + lane] = nd[x];
      }
      __syncwarp();
      // queries of this tile that may see this key: all of them, or (causal) those with q + off >= key
      const int q_first = p.causal ? max(0, krow - off - i * kW) : 0;  // first local query column that sees the key
      // Keys past the end need no mask (their rows of dK / dV are never stored and no other row depends on them);
      // only the causal diagonal does.
      {
        const float2 sl2 = make_float2(p.scale_log2, p.scale_log2), sc2 = make_float2(p.scale, p.scale);
        auto batch = [&](int col, const uint32_t (&rs)[16], const uint32_t (&rp)[16]) {
          uint32_t wp[8], wd[8];
          if (__all_sync(0xffffffffu, q_first <= col)) {
#pragma unroll
            for (int x = 0; x < 16; x += 4) {
              const float4 nl = *reinterpret_cast<const float4*>(slot + col + x);
              const float4 nd = *reinterpret_cast<const float4*>(slot + kW + col + x);
              const float2 e0 = __ffma2_rn(make_float2(__uint_as_float(rs[x]), __uint_as_float(rs[x + 1])), sl2,
                                           make_float2(nl.x, nl.y));
              const float2 e1 = __ffma2_rn(make_float2(__uint_as_float(rs[x + 2]), __uint_as_float(rs[x + 3])), sl2,
                                           make_float2(nl.z, nl.w));
              const float2 t0 = __ffma2_rn(make_float2(__uint_as_float(rp[x]), __uint_as_float(rp[x + 1])), sc2,
                                           make_float2(nd.x, nd.y));
              const float2 t1 = __ffma2_rn(make_float2(__uint_as_float(rp[x + 2]), __uint_as_float(rp[x + 3])), sc2,
                                           make_float2(nd.z, nd.w));
              const float2 p0 = make_float2(ex2f(e0.x), ex2f(e0.y)), p1 = make_float2(ex2f(e1.x), ex2f(e1.y));
              const float2 d0 = __fmul2_rn(p0, t0), d1 = __fmul2_rn(p1, t1);
              const __nv_bfloat162 a0 = __floats2bfloat162_rn(p0.x, p0.y), a1 = __floats2bfloat162_rn(p1.x, p1.y);
              const __nv_bfloat162 b0 = __floats2bfloat162_rn(d0.x, d0.y), b1 = __floats2bfloat162_rn(d1.x, d1.y);
              wp[x >> 1] = *reinterpret_cast<const uint32_t*>(&a0);
              wp[(x >> 1) + 1] = *reinterpret_cast<const uint32_t*>(&a1);
              wd[x >> 1] = *reinterpret_cast<const uint32_t*>(&b0);
              wd[(x >> 1) + 1] = *reinterpret_cast<const uint32_t*>(&b1);
            }
          } else {
#pragma unroll
            for (int x = 0; x < 16; x += 2) {
              float p0 = 0.f, p1 = 0.f, d0 = 0.f, d1 = 0.f;
              const int qa = col + x;
              if (qa >= q_first) {
                p0 = ex2f(fmaf(__uint_as_float(rs[x]), p.scale_log2, slot[qa]));
                d0 = p0 * fmaf(__uint_as_float(rp[x]), p.scale, slot[kW + qa]);
              }
              if (qa + 1 >= q_first) {
                p1 = ex2f(fmaf(__uint_as_float(rs[x + 1]), p.scale_log2, slot[qa + 1]));
                d1 = p1 * fmaf(__uint_as_float(rp[x + 1]), p.scale, slot[kW + qa + 1]);
              }
              const __nv_bfloat162 a = __floats2bfloat162_rn(p0, p1), d = __floats2bfloat162_rn(d0, d1);
              wp[x >> 1] = *reinterpret_cast<const uint32_t*>(&a);
              wd[x >> 1] = *reinterpret_cast<const uint32_t*>(&d);
            }
          }
          store_cols16(my_pt, row, col, wp);
          store_cols16(my_dst, row, col, wd);
        };
        walk_columns(t_s, t_s + kW, batch);
      }
      ptx::tc_fence_before();
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&pt_full[g]);
    }
    if (n_iter == 0 && krow < p.Skv && g == 0) {  // no query sees these keys
      __nv_bfloat16* dv = p.dv + ((static_cast<long long>(b) * p.Skv + krow) * p.H + h) * D;
      __nv_bfloat16* dk = p.dk + ((static_cast<long long>(b) * p.Skv + krow) * p.H + h) * D;
#pragma unroll
      for (int q = 0; q < D / 8; ++q) {
        reinterpret_cast<uint4*>(dv)[q] = make_uint4(0u, 0u, 0u, 0u);
        reinterpret_cast<uint4*>(dk)[q] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    if (n_iter > 0 && ok && g < 2) {  // all uniform over the warp
      const bool done = ptx::mbar_wait(acc_full, 0, abort_flag, p.timeout_ns);
      if (!__all_sync(0xffffffffu, done)) {
        if (lane == 0) report_status(p.status, kStatusGemmTimeout, 77, blockIdx.x, 0);
      } else {
        ptx::tc_fence_after();
        // one group stores the dV rows, the other the dK rows
        if (g == 0)
          store_row_bf16(p.dv + ((static_cast<long long>(b) * p.Skv + krow) * p.H + h) * D, t_dv + t_row,
                         krow < p.Skv, 0, D / 32);
        else
          store_row_bf16(p.dk + ((static_cast<long long>(b) * p.Skv + krow) * p.H + h) * D, t_dk + t_row,
                         krow < p.Skv, 0, D / 32);
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, kTmemBwd);
  }
}

// delta[b, h, s] = sum_d dO[b, s, h, d] * O[b, s, h, d]  (both [B, S, H, D] contiguous bf16); D / 8 lanes per row, 16 bytes
// of either operand each.  Bound by HBM (8 x 16 heads of 64, 1024 rows: a warp per row took 20.8 us; it added the row in another
// order, which moves the gradients by roundings of dS to bf16).
template <int D>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o, float* __restrict__ delta,
                  int B, int H, int S) {
  constexpr int kLanes = D / 8;
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x, row = i / kLanes;  // over B * S * H
  const bool in = row < static_cast<long long>(B) * S * H;
  float acc = 0.f;
  if (in) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(o) + i), g = __ldg(reinterpret_cast<const uint4*>(d_o) + i);
    const __nv_bfloat162 *av = reinterpret_cast<const __nv_bfloat162*>(&a), *gv = reinterpret_cast<const __nv_bfloat162*>(&g);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 x = __bfloat1622float2(av[k]), y = __bfloat1622float2(gv[k]);
      acc += x.x * y.x + x.y * y.y;
    }
  }
#pragma unroll
  for (int s = kLanes / 2; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (in && threadIdx.x % kLanes == 0) {
    const int hh = static_cast<int>(row % H);
    const long long bs = row / H;
    const int ss = static_cast<int>(bs % S);
    const long long bb = bs / S;
    delta[(bb * H + hh) * S + ss] = acc;
  }
}

typedef CUresult (*EncodeTiledFnB)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFnB encode_fn_b() {
  // The driver's encoder wants a current context; a thread that has made no runtime call yet (an autograd
  // worker entering its first backward) has none, and the encoder then fails with CUDA_ERROR_INVALID_CONTEXT.
  static thread_local bool bound = false;
  if (!bound) {  // cudaSetDevice binds the primary context to the thread and is legal during stream capture
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaSetDevice(dev);
    bound = true;
  }
  static EncodeTiledFnB fn = nullptr;
  if (fn == nullptr) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeTiledFnB>(sym);
  }
  return fn;
}

// [B, H, S, D] bf16 view with element strides (sb, sh, ss): 4-D map, 64 x `rows` x 1 x 1 box, rows past S read zeros.
int g_map_error = 0;  // why the last map_bhsd failed: -1 no driver entry point, -2 / -3 alignment, > 0 the driver's code

bool map_bhsd(CUtensorMap* map, const void* ptr, int B, int H, int S, int kD, long long sb, long long sh, long long ss,
              int rows) {
  EncodeTiledFnB enc = encode_fn_b();
  g_map_error = -1;
  if (enc == nullptr) return false;
  g_map_error = -2;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0 || ss % 8 || ss < kD) return false;
  g_map_error = -3;
  if ((H > 1 && (sh % 8 || sh <= 0)) || (B > 1 && (sb % 8 || sb <= 0))) return false;
  const long long sh_ok = H > 1 ? sh : ss * S + ((8 - (ss * S) % 8) % 8);
  const long long sb_ok = B > 1 ? sb : sh_ok * H;
  cuuint64_t dims[4] = {static_cast<cuuint64_t>(kD), static_cast<cuuint64_t>(S), static_cast<cuuint64_t>(H),
                        static_cast<cuuint64_t>(B)};
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(ss) * 2, static_cast<cuuint64_t>(sh_ok) * 2,
                           static_cast<cuuint64_t>(sb_ok) * 2};
  cuuint32_t box[4] = {64, static_cast<cuuint32_t>(rows), 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  g_map_error = static_cast<int>(enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides,
                                       box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
  return g_map_error == 0;
}

}  // namespace
}  // namespace fb

// Reason of the last -2 ... -5 of fb_attention_bwd (see g_map_error).
extern "C" int fb_attention_bwd_map_error() { return fb::g_map_error; }

namespace fb {
namespace {
template <int D>
int launch_bwd(const CUtensorMap (&fixed)[4], const CUtensorMap (&walked)[4], const void* out, const void* d_out, const BwdArgs& a, cudaStream_t stream) {
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(attn_bwd_dq_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             BwdCfg<D>::kSmemDq) != cudaSuccess ||
        cudaFuncSetAttribute(attn_bwd_dkv_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             BwdCfg<D>::kSmemDkv) != cudaSuccess)
      return static_cast<int>(cudaGetLastError());
    attr_set = true;
  }
  const long long rows = static_cast<long long>(a.B) * a.Sq * a.H;
  attn_delta_kernel<D><<<static_cast<unsigned>((rows * (D / 8) + 255) / 256), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(d_out),
      const_cast<float*>(a.delta), a.B, a.H, a.Sq);
  attn_bwd_dq_kernel<D><<<dim3((a.Sq + kT - 1) / kT, a.B * a.H), BwdCfg<D>::kThreads, BwdCfg<D>::kSmemDq, stream>>>(
      fixed[0], walked[1], walked[2], fixed[3], a);
  attn_bwd_dkv_kernel<D><<<dim3((a.Skv + kT - 1) / kT, a.B * a.H), BwdCfg<D>::kThreads, BwdCfg<D>::kSmemDkv, stream>>>(
      walked[0], fixed[1], fixed[2], walked[3], a);
  return static_cast<int>(cudaGetLastError());
}
}  // namespace
}  // namespace fb

// Gradients of out = softmax(scale q k^T) v (head dimension D = 64 or 128, bf16).  q, k, v: [B, H, S, D] views with
// element strides (last dimension contiguous, strides multiples of 8); out, d_out: [B, Sq, H, D] contiguous (the
// forward kernel's output layout); lse: [B, H, Sq] fp32 as written by fb_attention_fwd; delta: [B, H, Sq] fp32
// scratch that this call fills.  dq: [B, Sq, H, D], dk, dv: [B, Skv, H, D], contiguous bf16.  Returns -2 ... -5
// when q / k / v / d_out cannot be described by a TMA map.
extern "C" int fb_attention_bwd(const void* q, const void* k, const void* v, const void* out, const void* d_out,
                                const float* lse, float* delta, void* dq, void* dk, void* dv, int B, int H, int Sq,
                                int Skv, int D, long long q_sb, long long q_sh, long long q_ss, long long k_sb,
                                long long k_sh, long long k_ss, long long v_sb, long long v_sh, long long v_ss,
                                float scale, int causal, int32_t* status, cudaStream_t stream) {
  using namespace fb;
  if (B <= 0 || H <= 0 || Sq <= 0 || Skv <= 0 || (causal && Skv < Sq) || (D != 64 && D != 128)) return -1;
  if (lse == nullptr || delta == nullptr || out == nullptr || d_out == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv) |
       reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(d_out)) & 15)
    return -1;
  // q, k, v, d_out as the stationary side of a kernel (tiles of 128 rows) and as the side that is walked (64)
  CUtensorMap fixed[4], walked[4];
  const long long o_sb = static_cast<long long>(Sq) * H * D, o_sh = D, o_ss = static_cast<long long>(H) * D;
  for (auto [maps, rows] : {std::make_pair(fixed, kT), std::make_pair(walked, kW)}) {
    if (!map_bhsd(&maps[0], q, B, H, Sq, D, q_sb, q_sh, q_ss, rows)) return -2;
    if (!map_bhsd(&maps[1], k, B, H, Skv, D, k_sb, k_sh, k_ss, rows)) return -3;
    if (!map_bhsd(&maps[2], v, B, H, Skv, D, v_sb, v_sh, v_ss, rows)) return -4;
    if (!map_bhsd(&maps[3], d_out, B, H, Sq, D, o_sb, o_sh, o_ss, rows)) return -5;
  }
  BwdArgs a;
  a.dq = static_cast<__nv_bfloat16*>(dq);
  a.dk = static_cast<__nv_bfloat16*>(dk);
  a.dv = static_cast<__nv_bfloat16*>(dv);
  a.lse = lse;
  a.delta = delta;
  a.B = B;
  a.H = H;
  a.Sq = Sq;
  a.Skv = Skv;
  a.scale = scale;
  a.scale_log2 = scale * kLog2e;
  a.causal = causal ? 1 : 0;
  a.status = status;
  a.timeout_ns = 2000000000ull;
  return D == 64 ? launch_bwd<64>(fixed, walked, out, d_out, a, stream)
                 : launch_bwd<128>(fixed, walked, out, d_out, a, stream);
}
