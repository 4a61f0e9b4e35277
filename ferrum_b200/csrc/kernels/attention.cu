// Blockwise (flash-style) attention forward on the tcgen05 tensor cores, head dimension 64 or 128, bf16.
//
// The reference materialises the [S, S] score matrix per head on the host (ferrum-nn/src/transformer.rs:127-220).
// This kernel never writes scores to memory: one CTA owns two tiles of 128 query rows of one (batch, head) and walks
// the keys / values in tiles of 128:
//
//   warp 0       TMA producer: both Q tiles, then K_0, V_0, K_1, V_1, ... through one ring of tile-sized slots
//                (128-byte swizzle; a 128-wide head is two 64-column blocks per tile)
//   warp 1       one thread issues the MMAs: S = Q K_j^T (128 x 128 x D) into tensor memory, O_j = P_j V_j
//                (128 x D x 128) into a second region; both for either query tile
//   warps 4-7,   softmax of the first / second query tile: thread = query row.  Reads its row of S from tensor memory
//   warps 8-11   (tcgen05.ld), keeps the running maximum and sum (online softmax, base-2 exponentials), writes P_j as
//                bf16 into shared memory in the swizzled K-major layout the tensor core reads, and adds O_j-1 to its
//                accumulators in registers, rounded to nearest.
//
// What bounds it: the exponentials (16 per clock and SM: 2048 clocks per pair of tiles, as long as the MMAs of D = 128)
// and the instructions around them.  Hence the two query tiles: one group's exponentials run beside the other's
// reductions, and a group never waits for its own products: S_j+1 is issued as soon as S_j has left tensor memory
// (P_j is still being packed then), and O_j is picked up one tile later, when the next maximum is known.  16 heads of
// 128, 8192 rows, causal: 639 us with one query tile per CTA, where every tile paid both round trips to the tensor core;
// 340 with two, S_j+1 behind P_j and the MMA descriptors in ordinary registers, which made their issue the bound; now 288
// (950 TFLOP/s).  8 x 16 heads of 64, 1024 rows: 97, 88 and 84 us; 4 x 16 heads of 64, 8192 rows, causal: 1404, 973 and
// 923.  The same bits.
//
// Every mbarrier wait is bounded (status block + abort flag shared by the CTA's roles); nothing traps.
// Output: [B, S, H, D] contiguous bf16 (so the output projection sees [B, S, H*D]) and, optionally, the
// log-sum-exp of every row (natural log) for a recomputing backward.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../common/ptx.cuh"
#include "../common/status.h"
#include "../include/ferrum_kernels.h"

namespace fb {
namespace {

constexpr int kBQ = 128;          // query rows per group
constexpr int kBKV = 128;         // keys per tile
constexpr int kBlk = 128 * 128;   // 16 KB: 128 rows of 64 bf16 = one 128-byte-swizzled block
constexpr int kAttnThreads = 128 + 2 * kBQ;
// Registers: 168 a thread at launch (3 x 128 threads); the issuing warps keep 104 and the softmax warps, whose output
// row lives in registers, get 200: 104 + 200 + 200 = 3 x 168.
constexpr int kRegsIssue = 104, kRegsSoftmax = 200;
constexpr int kTmemColsAttn = 512;  // S of the groups: columns 0 and 128; O: 256 and 256 + D
// D = head dimension (64 or 128): an operand tile is D / 64 blocks side by side in the reduction (Q, K) or output (V)
// dimension; P is always 128 x 128 = two blocks.
template <int D>
struct AttnCfg {
  static constexpr int kNB = D / 64;
  static constexpr int kTile = kNB * kBlk;
  static constexpr int kRing = D == 64 ? 6 : 3;  // three 32 KB slots are what Q and P leave room for
  static constexpr int kBody = kTile * (2 + kRing) + 2 * 2 * kBlk;
  static constexpr int kSmem = kBody + 1024 + 256;
  static constexpr int kChunk = D == 64 ? 32 : 16;  // score columns per tensor-memory load (two in flight)
};

struct AttnArgs {
  __nv_bfloat16* out;   // [B, Sq, H, D]
  float* lse;           // [B, H, Sq] or NULL
  int B, H, Sq, Skv;
  float scale_log2;     // softmax scale * log2(e)
  int causal;           // 1: query i attends keys j <= i + (Skv - Sq) (needs Skv >= Sq)
  int groups;           // query tiles per CTA (1: the second group idles)
  int q_blocks, head_group;
  int32_t* status;
  unsigned long long timeout_ns;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 fma2(float2 x, float2 y, float2 z) {
  float2 r;
  asm("{\n.reg .b64 a, b, c, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %7};\n"
      "fma.rn.f32x2 d, a, b, c;\nmov.b64 {%0, %1}, d;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y), "f"(z.x), "f"(z.y));
  return r;
}
// (x + y) * s, both rounded.  (As x * s + y it would be one operation less in the loop, but a packed product and sum are
// contracted to a multiply-add, other bits.)
__device__ __forceinline__ float2 add_scale2(float2 x, float2 y, float2 s) {
  float2 r;
  asm("{\n.reg .b64 a, b, c, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %7};\n"
      "add.rn.f32x2 d, a, b;\nmul.rn.f32x2 d, d, c;\nmov.b64 {%0, %1}, d;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y), "f"(s.x), "f"(s.y));
  return r;
}
__device__ __forceinline__ void tmem_ld(uint32_t addr, uint32_t (&r)[16]) { ptx::tmem_ld_32x32b_x16(addr, r); }
__device__ __forceinline__ void tmem_ld(uint32_t addr, uint32_t (&r)[32]) { ptx::tmem_ld_32x32b_x32(addr, r); }
// A store that may move across the waits for tensor memory (the fence in front of the arrival keeps it before that).
__device__ __forceinline__ void st_shared(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d));
}
// Waits for the loads in flight; the registers pass through, so that no use of them can move above the wait.
template <int N>
__device__ __forceinline__ void tmem_ready(uint32_t (&r)[N]) {
  ptx::tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < N; i += 16)
    asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]),
                      "+r"(r[i + 6]), "+r"(r[i + 7]), "+r"(r[i + 8]), "+r"(r[i + 9]), "+r"(r[i + 10]), "+r"(r[i + 11]),
                      "+r"(r[i + 12]), "+r"(r[i + 13]), "+r"(r[i + 14]), "+r"(r[i + 15]));
}

// Row maximum of the raw scores over the first `valid` columns (the scale is positive, applied once afterwards).
template <int CH, bool kMask>
__device__ __forceinline__ float row_max(uint32_t t_s, int valid) {
  constexpr int kN = kBKV / CH;
  uint32_t r[2][CH];
  float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  tmem_ld(t_s, r[0]);
#pragma unroll
  for (int c = 0; c < kN; ++c) {
    tmem_ready(r[c & 1]);
    if (c + 1 < kN) tmem_ld(t_s + (c + 1) * CH, r[(c + 1) & 1]);
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const float v = __uint_as_float(r[c & 1][i]);
      if (!kMask || c * CH + i < valid) mx[i & 3] = fmaxf(mx[i & 3], v);
    }
  }
  return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
}

// p = 2^(s * scale - m): adds the row sum to l, 32 columns at a time, and writes bf16 P into shared memory (K-major,
// 128-byte swizzle).  One warp of a group per scheduler: a chunk's exponentials are started before the chunk ahead is
// added up, packed and stored, so that the unit that evaluates them does not wait for that.  `s_read` runs when the last
// scores have left tensor memory.
template <int CH, bool kMask, typename F>
__device__ __forceinline__ void row_exp(uint32_t t_s, int valid, float scale, float neg_m, uint8_t* sp, int row,
                                        float& l, F&& s_read) {
  constexpr int kN = kBKV / CH;
  uint32_t r[2][CH];
  float2 e[2][CH / 2];
  float part = 0.f;
  const float2 sc = make_float2(scale, scale), nm = make_float2(neg_m, neg_m);
  tmem_ld(t_s, r[0]);
#pragma unroll
  for (int c = 0; c <= kN; ++c) {
    if (c < kN) {
      tmem_ready(r[c & 1]);
      if (c + 1 < kN) tmem_ld(t_s + (c + 1) * CH, r[(c + 1) & 1]);
      else s_read();
#pragma unroll
      for (int i = 0; i < CH; i += 2) {
        const float2 x = fma2(make_float2(__uint_as_float(r[c & 1][i]), __uint_as_float(r[c & 1][i + 1])), sc, nm);
        e[c & 1][i / 2] = make_float2(ex2(x.x), ex2(x.y));
      }
    }
    if (c == 0) continue;
    const int d = c - 1;
    uint32_t packed[CH / 2];
#pragma unroll
    for (int i = 0; i < CH; i += 2) {
      float2 v = e[d & 1][i / 2];
      if (kMask) {
        if (d * CH + i >= valid) v.x = 0.f;
        if (d * CH + i + 1 >= valid) v.y = 0.f;
      }
      part += v.x + v.y;
      const __nv_bfloat162 pk = __floats2bfloat162_rn(v.x, v.y);
      packed[i >> 1] = *reinterpret_cast<const uint32_t*>(&pk);
    }
    if ((d + 1) * CH % 32 == 0) {
      l += part;
      part = 0.f;
    }
    const uint32_t blk = ptx::smem_u32(sp) + (d * CH / 64) * kBlk + row * 128;
#pragma unroll
    for (int q = 0; q < CH / 8; ++q) {
      const int chunk = (d * CH % 64) / 8 + q;
      st_shared(blk + ((chunk ^ (row & 7)) << 4), packed[q * 4], packed[q * 4 + 1], packed[q * 4 + 2], packed[q * 4 + 3]);
    }
  }
}

template <int D>
__global__ void __launch_bounds__(kAttnThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const AttnArgs p) {
  using C = AttnCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int kNB = C::kNB, kTileBytes = C::kTile, kRing = C::kRing, kChunk = C::kChunk;
  uint8_t* sq = smem;                          // one tile per group
  uint8_t* ring = sq + 2 * kTileBytes;         // K_0, V_0, K_1, V_1, ... : item i in slot i % kRing
  uint8_t* sp = ring + kRing * kTileBytes;     // P of the groups: two k-blocks of 128 rows x 128 bytes each
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + C::kBody);
  uint64_t* full = q_full + 1;       // [kRing]
  uint64_t* empty = full + kRing;    // [kRing]
  uint64_t* s_full = empty + kRing;  // [2]
  uint64_t* s_free = s_full + 2;     // [2]
  uint64_t* p_full = s_free + 2;     // [2]
  uint64_t* o_full = p_full + 2;     // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  // CTAs in the order of `head_group` heads at a time (their keys and values stay in L2), the query blocks with the
  // most keys first: under a causal mask the short ones fill the end of the last wave.
  const int t = static_cast<int>(blockIdx.x), per_group = p.head_group * p.q_blocks;
  const int first = (t / per_group) * p.head_group, heads = min(p.head_group, p.B * p.H - first);
  const int rest = t - first * p.q_blocks;
  const int bh = first + rest % heads, qb = p.q_blocks - 1 - rest / heads;
  const int h = bh % p.H, b = bh / p.H;
  const int q0 = qb * p.groups * kBQ;
  // causal: a tile's last query row bounds the keys any of its rows may see
  int n[2];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const int row0 = q0 + g * kBQ;
    const int kv_end = p.causal ? min(p.Skv, row0 + kBQ + (p.Skv - p.Sq)) : p.Skv;
    n[g] = g < p.groups && row0 < p.Sq ? (kv_end + kBKV - 1) / kBKV : 0;
  }
  const int n_max = max(n[0], n[1]);

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    ptx::mbar_init(q_full, 1);
    for (int s = 0; s < kRing; ++s) {
      ptx::mbar_init(&full[s], 1);
      ptx::mbar_init(&empty[s], 1);
    }
    for (int g = 0; g < 2; ++g) {
      ptx::mbar_init(&s_full[g], 1);
      ptx::mbar_init(&s_free[g], 4);  // one arrival per softmax warp
      ptx::mbar_init(&p_full[g], 4);
      ptx::mbar_init(&o_full[g], 1);
    }
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&map_q);
    ptx::prefetch_tensormap(&map_k);
    ptx::prefetch_tensormap(&map_v);
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, kTmemColsAttn);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
    if (warp == 0 && lane == 0) {
      // ---------------------------------------------------------------- TMA producer
      const int q_tiles = (n[0] > 0) + (n[1] > 0);
      ptx::mbar_arrive_expect_tx(q_full, q_tiles * kTileBytes);
      for (int g = 0; g < q_tiles; ++g)
#pragma unroll
        for (int nb = 0; nb < kNB; ++nb)
          ptx::tma_load_4d(sq + g * kTileBytes + nb * kBlk, &map_q, q_full, nb * 64, q0 + g * kBQ, h, b);
      int issued = 0;
      for (; issued < 2 * n_max; ++issued) {
        const int s = issued % kRing;
        if (!ptx::mbar_wait(&empty[s], ((issued / kRing) & 1) ^ 1, abort_flag, p.timeout_ns)) {
          report_status(p.status, kStatusGemmTimeout, 51, blockIdx.x, issued);
          break;
        }
        ptx::mbar_arrive_expect_tx(&full[s], kTileBytes);
        const void* map = (issued & 1) ? static_cast<const void*>(&map_v) : static_cast<const void*>(&map_k);
#pragma unroll
        for (int nb = 0; nb < kNB; ++nb)
          ptx::tma_load_4d(ring + s * kTileBytes + nb * kBlk, map, &full[s], nb * 64, (issued >> 1) * kBKV, h, b);
      }
      if (issued < 2 * n_max || *abort_flag) {  // given up: no copy may outlive the CTA (bounded)
        const uint64_t t0 = ptx::globaltimer();
        while (!ptx::mbar_try_wait(q_full, 0) && ptx::globaltimer() - t0 <= p.timeout_ns) {
        }
        for (int s = 0; s < kRing && s < issued; ++s)
          while (!ptx::mbar_try_wait(&full[s], ((issued - 1 - s) / kRing) & 1) &&
                 ptx::globaltimer() - t0 <= p.timeout_ns) {
          }
      }
    } else if (warp == 1 && ptx::elect_one()) {
      // ---------------------------------------------------------------- MMA issuer
      const uint32_t idesc_s = ptx::make_idesc(1u, kBQ, kBKV, 0, 0);   // Q, K both K-major
      const uint32_t idesc_o = ptx::make_idesc(1u, kBQ, D, 0, 1);      // P K-major, V with d contiguous (MN-major)
      const uint64_t q_first = ptx::make_smem_desc_sw128(ptx::smem_u32(sq), 16, 1024);
      const uint64_t ring_first = ptx::make_smem_desc_sw128(ptx::smem_u32(ring), 16, 1024);
      const uint64_t v_first = ptx::make_smem_desc_sw128(ptx::smem_u32(ring), kBlk, 1024);
      const uint64_t p_first = ptx::make_smem_desc_sw128(ptx::smem_u32(sp), 16, 1024);
      auto wait_item = [&](int i) { return ptx::mbar_wait(&full[i % kRing], (i / kRing) & 1, abort_flag, p.timeout_ns); };
      auto last_of = [&](int j) { return j < n[1] ? 1 : 0; };  // the group that uses tile j last
      auto issue_s = [&](int g, int j) {
        const uint64_t a = ptx::desc_advance(q_first, g * kTileBytes), b = ptx::desc_advance(ring_first, (2 * j % kRing) * kTileBytes);
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          ptx::umma_f16(tmem_base + g * kBKV, ptx::desc_advance(a, (k >> 2) * kBlk + (k & 3) * 32),
                        ptx::desc_advance(b, (k >> 2) * kBlk + (k & 3) * 32), idesc_s, k != 0 ? 1u : 0u);
        ptx::umma_commit(&s_full[g]);
        if (g == last_of(j)) ptx::umma_commit(&empty[2 * j % kRing]);  // free once these MMAs have read it
      };
      auto issue_o = [&](int g, int j) {
        const uint64_t a = ptx::desc_advance(p_first, g * 2 * kBlk), b = ptx::desc_advance(v_first, (2 * j + 1) % kRing * kTileBytes);
#pragma unroll
        for (int k = 0; k < kBKV / 16; ++k)
          // V: 16 keys (rows of 128 bytes) per MMA; its 64-column blocks lie kBlk apart (the leading-dimension offset)
          ptx::umma_f16(tmem_base + 2 * kBKV + g * D, ptx::desc_advance(a, (k >> 2) * kBlk + (k & 3) * 32),
                        ptx::desc_advance(b, k * 2048), idesc_o, k != 0 ? 1u : 0u);
        ptx::umma_commit(&o_full[g]);
        if (g == last_of(j)) ptx::umma_commit(&empty[(2 * j + 1) % kRing]);
      };
      bool ok = ptx::mbar_wait(q_full, 0, abort_flag, p.timeout_ns) && wait_item(0);
      if (!ok) report_status(p.status, kStatusGemmTimeout, 52, blockIdx.x, 0);
      if (ok) {
        ptx::tc_fence_after();
        for (int g = 0; g < 2; ++g)
          if (n[g] > 0) issue_s(g, 0);
      }
      for (int j = 0; ok && j < n_max; ++j) {
        for (int g = 0; ok && g < 2; ++g) {
          if (j >= n[g]) continue;
          if (j + 1 < n[g]) {  // S_j has been read
            ok = ptx::mbar_wait(&s_free[g], j & 1, abort_flag, p.timeout_ns) && wait_item(2 * (j + 1));
            if (ok) {
              ptx::tc_fence_after();
              issue_s(g, j + 1);
            }
          }
          // P_j is written and O_(j-1) picked up
          ok = ok && ptx::mbar_wait(&p_full[g], j & 1, abort_flag, p.timeout_ns) && wait_item(2 * j + 1);
          if (!ok) {
            report_status(p.status, kStatusGemmTimeout, 53, blockIdx.x, j);
            break;
          }
          ptx::tc_fence_after();
          issue_o(g, j);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
    // ------------------------------------------------------------------ softmax + output (thread = query row)
    const int g = (warp - 4) >> 2, quarter = warp & 3;
    const int row = quarter * 32 + lane, q_row = q0 + g * kBQ + row, n_tiles = g ? n[1] : n[0];
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t t_s = lane_base + g * kBKV, t_o = lane_base + 2 * kBKV + g * D;
    uint8_t* my_p = sp + g * 2 * kBlk;
    float m = -INFINITY, l = 0.f;
    float2 o[D / 2];
#pragma unroll
    for (int i = 0; i < D / 2; ++i) o[i] = make_float2(0.f, 0.f);
    bool ok = n_tiles > 0;
    auto wait_all = [&](uint64_t* bar, int phase, int code, int j) {
      const bool ready = ptx::mbar_wait(bar, phase, abort_flag, p.timeout_ns);
      if (__all_sync(0xffffffffu, ready)) {
        ptx::tc_fence_after();
        return true;
      }
      if (lane == 0) report_status(p.status, kStatusGemmTimeout, code, blockIdx.x, j);
      return false;
    };
    auto add_o = [&](float scale) {  // o = (o + the product of the tile before) * scale
      const float2 sc = make_float2(scale, scale);
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t r[32];
        tmem_ld(t_o + c * 32, r);
        tmem_ready(r);
#pragma unroll
        for (int i = 0; i < 16; ++i)
          o[c * 16 + i] = add_scale2(o[c * 16 + i], make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), sc);
      }
    };
    auto s_read = [&]() {
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&s_free[g]);
    };
    for (int j = 0; j < n_tiles; ++j) {
      ok = wait_all(&s_full[g], j & 1, 55, j);
      if (!ok) break;
      int valid = min(kBKV, p.Skv - j * kBKV);  // columns past it are padding
      if (p.causal) valid = max(0, min(valid, q_row + (p.Skv - p.Sq) + 1 - j * kBKV));  // this row's keys only
      // (0 is possible from the second tile on — all of the row's keys lie in earlier tiles — and harmless: the
      // running maximum is finite by then, so alpha = 1 and every p = 0; the first tile always holds key 0)
      const bool whole = __all_sync(0xffffffffu, valid == kBKV);
      const float mx = whole ? row_max<kChunk, false>(t_s, valid) : row_max<kChunk, true>(t_s, valid);
      const float m_new = fmaxf(m, mx * p.scale_log2);
      const float alpha = ex2(m - m_new);  // 0 for the first tile (m = -inf)
      m = m_new;
      if (j > 0) {  // O_(j-1): its accumulators are free and its P has been read
        ok = wait_all(&o_full[g], (j - 1) & 1, 56, j);
        if (!ok) break;
        add_o(alpha);
      }
      l = __fmul_rn(l, alpha);
      if (whole)
        row_exp<kChunk, false>(t_s, valid, p.scale_log2, -m, my_p, row, l, s_read);
      else
        row_exp<kChunk, true>(t_s, valid, p.scale_log2, -m, my_p, row, l, s_read);
      ptx::tc_fence_before();          // the reads of S and O are ordered before the MMAs that overwrite them
      ptx::fence_proxy_async_smem();   // P becomes visible to the tensor core's (async-proxy) reads
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&p_full[g]);
    }
    if (ok) ok = wait_all(&o_full[g], (n_tiles - 1) & 1, 57, n_tiles);
    if (ok) add_o(1.f);
    if (ok && q_row < p.Sq) {
      const float inv = 1.f / l;
      __nv_bfloat16* dst = p.out + ((static_cast<long long>(b) * p.Sq + q_row) * p.H + h) * D;
#pragma unroll
      for (int q = 0; q < D / 8; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __nv_bfloat162 pk = __floats2bfloat162_rn(o[q * 4 + e].x * inv, o[q * 4 + e].y * inv);
          w[e] = *reinterpret_cast<const uint32_t*>(&pk);
        }
        reinterpret_cast<uint4*>(dst)[q] = make_uint4(w[0], w[1], w[2], w[3]);
      }
      if (p.lse != nullptr)
        p.lse[(static_cast<long long>(b) * p.H + h) * p.Sq + q_row] = (m + log2f(l)) * 0.6931471805599453f;
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, kTmemColsAttn);
  }
}

int attn_sm_count() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}

typedef CUresult (*EncodeTiledFnA)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFnA encode_fn_a() {
  // The driver's encoder wants a current context; a thread that has made no runtime call yet (an autograd
  // worker entering its first backward) has none, and the encoder then fails with CUDA_ERROR_INVALID_CONTEXT.
  static thread_local bool bound = false;
  if (!bound) {  // cudaSetDevice binds the primary context to the thread and is legal during stream capture
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaSetDevice(dev);
    bound = true;
  }
  static EncodeTiledFnA fn = nullptr;
  if (fn == nullptr) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeTiledFnA>(sym);
  }
  return fn;
}

// [B, H, S, D] bf16 view with element strides (sb, sh, ss), last dimension contiguous: a 4-D map with a
// 64 x 128 x 1 x 1 box (one 64-column block of 128 rows); rows past S read zeros.
bool make_map_bhsd(CUtensorMap* map, const void* ptr, int B, int H, int S, int kD, long long sb, long long sh,
                   long long ss) {
  EncodeTiledFnA enc = encode_fn_a();
  if (enc == nullptr) return false;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0 || ss % 8 || ss < kD) return false;
  if ((H > 1 && (sh % 8 || sh <= 0)) || (B > 1 && (sb % 8 || sb <= 0))) return false;
  // a dimension of extent 1 still needs a legal stride
  const long long sh_ok = H > 1 ? sh : ss * S + ((8 - (ss * S) % 8) % 8);
  const long long sb_ok = B > 1 ? sb : sh_ok * H;
  cuuint64_t dims[4] = {static_cast<cuuint64_t>(kD), static_cast<cuuint64_t>(S), static_cast<cuuint64_t>(H),
                        static_cast<cuuint64_t>(B)};
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(ss) * 2, static_cast<cuuint64_t>(sh_ok) * 2,
                           static_cast<cuuint64_t>(sb_ok) * 2};
  cuuint32_t box[4] = {64, 128, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int D>
int launch_attn(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, AttnArgs& a, cudaStream_t stream) {
  static const cudaError_t configured = cudaFuncSetAttribute(
      attn_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnCfg<D>::kSmem);
  if (configured != cudaSuccess) return static_cast<int>(configured);
  const long long heads = static_cast<long long>(a.B) * a.H, q_tiles = (a.Sq + kBQ - 1) / kBQ;
  // One query tile per CTA while every tile has an SM of its own, else two.
  a.groups = heads * q_tiles <= attn_sm_count() ? 1 : 2;
  a.q_blocks = static_cast<int>((q_tiles + a.groups - 1) / a.groups);
  // Heads whose keys and values fill half of L2 (but at least 16) go first, all query blocks of theirs, then the next.
  const long long fit = (64ll << 20) / (static_cast<long long>(a.Skv) * D * 4);
  const long long want = fit < 16 ? 16 : fit;
  a.head_group = static_cast<int>(want < heads ? want : heads);
  const long long grid = heads * a.q_blocks;
  if (grid > 0x7fffffffll) return -1;
  attn_fwd_kernel<D><<<static_cast<unsigned>(grid), kAttnThreads, AttnCfg<D>::kSmem, stream>>>(mq, mk, mv, a);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace
}  // namespace fb

// out[b, s, h, :] = softmax(scale * q[b,h,s,:] . k[b,h,:,:]^T) v[b,h,:,:]  for head dimension D = 64 or 128, bf16
// operands given as [B, H, S, D] views with element strides (last dimension contiguous, strides multiples of 8).
// out is [B, Sq, H, D] contiguous; lse (optional) [B, H, Sq] fp32.  Returns -2 when an operand cannot be described
// by a TMA map.  causal: query i sees keys j <= i + (Skv - Sq); key tiles past the diagonal are skipped.
extern "C" int fb_attention_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int B, int H,
                                int Sq, int Skv, int D, long long q_sb, long long q_sh, long long q_ss,
                                long long k_sb, long long k_sh, long long k_ss, long long v_sb, long long v_sh,
                                long long v_ss, float scale, int causal, int32_t* status, cudaStream_t stream) {
  using namespace fb;
  if (B <= 0 || H <= 0 || Sq <= 0 || Skv <= 0 || (causal && Skv < Sq) || (D != 64 && D != 128)) return -1;
  if (reinterpret_cast<uintptr_t>(out) & 15) return -1;
  CUtensorMap mq, mk, mv;
  if (!make_map_bhsd(&mq, q, B, H, Sq, D, q_sb, q_sh, q_ss) || !make_map_bhsd(&mk, k, B, H, Skv, D, k_sb, k_sh, k_ss) ||
      !make_map_bhsd(&mv, v, B, H, Skv, D, v_sb, v_sh, v_ss))
    return -2;
  AttnArgs a;
  a.out = static_cast<__nv_bfloat16*>(out);
  a.lse = lse;
  a.B = B;
  a.H = H;
  a.Sq = Sq;
  a.Skv = Skv;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.causal = causal ? 1 : 0;
  a.status = status;
  a.timeout_ns = 2000000000ull;
  return D == 64 ? launch_attn<64>(mq, mk, mv, a, stream) : launch_attn<128>(mq, mk, mv, a, stream);
}
