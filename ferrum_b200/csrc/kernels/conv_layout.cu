// Layout changes around the implicit-GEMM convolution (csrc/gemm/tcgen05_gemm.cu, fb_conv_igemm): the reference
// keeps activations as NCHW fp32 (ferrum-nn/src/conv.rs:209-330); the tensor-core kernels read NHWC bf16 through
// 4-D TMA boxes, with the channel count padded to a multiple of 8 so that every pixel starts on a 16-byte boundary.
//
// A convolution of any stride is one of stride 1 over a space-to-depth arrangement of its input:
//   z[b, I, J, (rh * ew + rw) * C + c] = x[b, c, I * sh + rh - ph, J * sw + rw - pw],  rh < eh = min(sh, kh), rw < ew,
// zero outside the image, with ceil(kh / sh) x ceil(kw / sw) filters (taps past kh x kw are zeros: an infinity in x makes
// NaN of the windows that only they reach).  Rows and columns that the stride skips altogether
// (kernel < stride: the 1 x 1 shortcut of a residual block) are not in z.  Stride 1 is the case sh = sw = 1, ph = pw = 0:
// a plain NCHW -> NHWC conversion, the padding being the TMA unit's zero fill.
//
//   fb_conv_pack_input    x -> z, optionally with the gradient of a ReLU in front (x counts where mask > 0)
//   fb_conv_pack_filters  [O, C, kh, kw] fp32 -> the bf16 filters of the forward product or of the data gradient
//   fb_conv_fold_wgrad    the splits of fb_conv_wgrad -> their sum as [O, C, kh, kw]
//   fb_s2d_nhwc_to_nchw_f32  the data gradient of z -> that of x
//   fb_nhwc_to_nchw_f32      a result [B, P, ld] -> [B, C, P], plus a residual, behind a ReLU
//   fb_nhwc_to_nchw_masks, fb_conv_pack_masked  the same with the ReLU's mask as bytes: a quarter of what its result is
//
// All are bound by HBM if they do not spend too many instructions: a pixel a load and store they were bound by their issue
// (ncu: 63 - 79 % of the slots, 23 - 39 % of the HBM rate), so rows of whole quads move four pixels at a time.  A residual
// block's step (64 images, 64 -> 128 channels, 56 x 56, stride 2), us before and after: 64 x 56 x 56 images to s2d 19.6 -
// 24 / 14.6, a gradient of 128 x 28 x 28 9.3 / 7.9, a result to NCHW 12.4 / 8.9.
// The input conversion goes through shared memory in blocks of 64 channels x 64 pixels of bf16
// pairs: 16-byte reads along the pixels, 16-byte writes along the channels.  (Results stored as NCHW from the GEMM's
// accumulator rows, a 4-byte store per channel and pixel, were slower than the transposing kernel: 243 us of GEMMs in a
// residual block's training step against 176 + 67.)
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../include/ferrum_kernels.h"

namespace fb {
namespace {

// A convolution as the layouts see it; q counts the columns of z times ew, r its rows times eh.
struct S2d {
  int C, H, W, sh, sw, eh, ew, ph, pw, Hz, Wz;
  long long ld;  // channels per pixel of the NHWC side (>= eh * ew * C)
};

constexpr int kTileC = 64, kTileQ = 64;

// Four values of a mask: floats, or bytes that say where.
__device__ __forceinline__ float4 mask4(const float* m) { return __ldg(reinterpret_cast<const float4*>(m)); }
__device__ __forceinline__ float4 mask4(const uint8_t* m) {
  const uchar4 u = __ldg(reinterpret_cast<const uchar4*>(m));
  return make_float4(u.x, u.y, u.z, u.w);
}

// kQuads: four pixels a load (rows of whole quads on 16-byte boundaries, no columns skipped).
template <bool kVec, bool kQuads, typename M>
__global__ void __launch_bounds__(256)
pack_input_kernel(const float* __restrict__ x, const M* __restrict__ mask, __nv_bfloat16* __restrict__ z, const S2d g,
                  int q_tiles) {
  __shared__ uint32_t tile[kTileC / 2][kTileQ + 1];
  const int q0 = static_cast<int>(blockIdx.x % q_tiles) * kTileQ;
  const long long br = blockIdx.x / q_tiles;
  const int rows = g.Hz * g.eh;
  const long long b = br / rows;
  const int r = static_cast<int>(br - b * rows), I = r / g.eh, rh = r - I * g.eh, i = I * g.sh + rh - g.ph;
  const int c0 = blockIdx.y * kTileC, nc = min(kTileC, g.C - c0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool row_in = i >= 0 && i < g.H;
  const long long plane = static_cast<long long>(g.H) * g.W;
  const long long base = (b * g.C + c0) * plane + static_cast<long long>(i) * g.W;
  const int n_q = g.Wz * g.ew;
  if constexpr (kQuads) {
    const int j_lo = q0 - g.pw, quad = threadIdx.x & 15, pair0 = threadIdx.x >> 4;  // j_lo: column of the tile's first pixel
    for (int j = (j_lo & ~3) + quad * 4; j < j_lo + kTileQ; j += 64) {
      const bool in = row_in && j >= 0 && j < g.W;  // a quad is inside or outside as a whole
      float4 v[2][2], m[2][2];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = (pair0 + 16 * k) * 2 + e;
          v[k][e] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (in && c < nc) v[k][e] = __ldg(reinterpret_cast<const float4*>(x + base + c * plane + j));
        }
      if (mask != nullptr) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int c = (pair0 + 16 * k) * 2 + e;
            m[k][e] = make_float4(1.f, 1.f, 1.f, 1.f);
            if (in && c < nc) m[k][e] = mask4(mask + base + c * plane + j);
          }
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (!(m[k][e].x > 0.f)) v[k][e].x = 0.f;
            if (!(m[k][e].y > 0.f)) v[k][e].y = 0.f;
            if (!(m[k][e].z > 0.f)) v[k][e].z = 0.f;
            if (!(m[k][e].w > 0.f)) v[k][e].w = 0.f;
          }
      }
      const int at = j - j_lo;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float4 a = v[k][0], b2 = v[k][1];
        const __nv_bfloat162 p[4] = {__floats2bfloat162_rn(a.x, b2.x), __floats2bfloat162_rn(a.y, b2.y),
                                     __floats2bfloat162_rn(a.z, b2.z), __floats2bfloat162_rn(a.w, b2.w)};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (at + e >= 0 && at + e < kTileQ) tile[pair0 + 16 * k][at + e] = *reinterpret_cast<const uint32_t*>(&p[e]);
      }
    }
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int q = q0 + h * 32 + lane;
      int j = q;
      if (g.sw != 1 || g.ew != 1) {
        const int J = q / g.ew;
        j = J * g.sw + q - J * g.ew;
      }
      j -= g.pw;
      const bool in = row_in && q < n_q && j >= 0 && j < g.W;
      float v[2][kTileC / 16];
#pragma unroll
      for (int k = 0; k < kTileC / 16; ++k) {
        const int c = (warp + 8 * k) * 2;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          v[e][k] = 0.f;
          if (in && c + e < nc) v[e][k] = __ldg(x + base + (c + e) * plane + j);
        }
      }
      if (mask != nullptr) {
#pragma unroll
        for (int k = 0; k < kTileC / 16; ++k) {
          const int c = (warp + 8 * k) * 2;
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (in && c + e < nc && !(static_cast<float>(__ldg(mask + base + (c + e) * plane + j)) > 0.f)) v[e][k] = 0.f;
        }
      }
#pragma unroll
      for (int k = 0; k < kTileC / 16; ++k) {
        const __nv_bfloat162 p = __floats2bfloat162_rn(v[0][k], v[1][k]);
        tile[warp + 8 * k][h * 32 + lane] = *reinterpret_cast<const uint32_t*>(&p);
      }
    }
  }
  __syncthreads();
  const int oct = threadIdx.x & 7;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int ql = k * 32 + (threadIdx.x >> 3), q = q0 + ql;
    if (q >= n_q) continue;
    const int J = q / g.ew, rw = q - J * g.ew;
    __nv_bfloat16* pixel = z + ((b * g.Hz + I) * g.Wz + J) * g.ld;
    __nv_bfloat16* dst = pixel + static_cast<long long>(rh * g.ew + rw) * g.C + c0 + oct * 8;
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = tile[oct * 4 + e][ql];
    if (kVec) {  // whole octets of channels on 16-byte boundaries; the tile holds zeros behind the last channel
      if (oct * 8 < nc) *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (oct * 8 + e < nc)
          dst[e] = __ushort_as_bfloat16(static_cast<unsigned short>(e & 1 ? w[e >> 1] >> 16 : w[e >> 1] & 0xffff));
      if (oct == 0 && c0 == 0 && rh == g.eh - 1 && rw == g.ew - 1)  // the padding channels
        for (long long c = static_cast<long long>(g.eh) * g.ew * g.C; c < g.ld; ++c) pixel[c] = __float2bfloat16_rn(0.f);
    }
  }
}

// Filter tap of channel ch of z under tap (I, J) of the stride-1 convolution; -1: there is none (a zero).
struct Filter {
  int O, C, kh, kw, sh, sw, eh, ew, k2h, k2w, pitch;  // pitch: elements per tap of a packed row
};
__device__ __forceinline__ int filter_at(const Filter& f, int I, int J, int ch, int& c) {
  const int rc = ch / f.C, rh = rc / f.ew, rw = rc - rh * f.ew;
  c = ch - rc * f.C;
  const int ki = I * f.sh + rh, kj = J * f.sw + rw;
  return rh < f.eh && ki < f.kh && kj < f.kw ? ki * f.kw + kj : -1;
}

// kDgrad = false: out[o][I, J][ch] (pitch >= eh ew C); true: out[ch][I, J flipped][o] (pitch >= O).  Index: int, or 64
// bits for filters beyond that.
template <bool kDgrad, typename Index>
__global__ void __launch_bounds__(256)
pack_filters_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ out, const Filter f, Index total) {
  for (Index at = blockIdx.x * 256 + threadIdx.x; at < total; at += gridDim.x * 256) {
    const Index rt = at / f.pitch;
    const int k = static_cast<int>(at - rt * f.pitch), taps = f.k2h * f.k2w, row = static_cast<int>(rt / taps);
    int tap = static_cast<int>(rt - static_cast<Index>(row) * taps);
    if (kDgrad) tap = taps - 1 - tap;
    const int I = tap / f.k2w, J = tap - I * f.k2w, ch = kDgrad ? row : k, o = kDgrad ? k : row;
    int c;
    const int t = filter_at(f, I, J, ch, c);
    const bool in = t >= 0 && o < f.O;
    out[at] = __float2bfloat16_rn(in ? __ldg(w + (static_cast<long long>(o) * f.C + c) * f.kh * f.kw + t) : 0.f);
  }
}

// dw[o, c, ki, kj] = sum over the splits of part[split][o][I, J][ch], in their order.
template <typename Index>
__global__ void __launch_bounds__(256)
fold_wgrad_kernel(const float* __restrict__ part, float* __restrict__ dw, const Filter f, int splits, Index total) {
  for (Index at = blockIdx.x * 256 + threadIdx.x; at < total; at += gridDim.x * 256) {
    const Index rt = at / f.pitch;
    const int ch = static_cast<int>(at - rt * f.pitch), taps = f.k2h * f.k2w, o = static_cast<int>(rt / taps);
    const int tap = static_cast<int>(rt - static_cast<Index>(o) * taps), I = tap / f.k2w, J = tap - I * f.k2w;
    int c;
    const int t = filter_at(f, I, J, ch, c);
    if (t < 0) continue;
    float s = 0.f;
#pragma unroll 8
    for (int i = 0; i < splits; ++i) s += __ldg(part + static_cast<long long>(i) * total + at);
    dw[(static_cast<long long>(o) * f.C + c) * f.kh * f.kw + t] = s;
  }
}

__global__ void __launch_bounds__(256)
s2d_to_nchw_kernel(const float* __restrict__ z, const float* __restrict__ add, float* __restrict__ x, const S2d g) {
  __shared__ float tile[32][33];
  const long long bi = blockIdx.x;
  const long long b = bi / g.H;
  const int i = static_cast<int>(bi - b * g.H);
  const int I = (i + g.ph) / g.sh, rh = (i + g.ph) % g.sh;
  const int j0 = blockIdx.y * 32, c0 = blockIdx.z * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int j = j0 + ty + 8 * k, c = c0 + tx;
    float v = 0.f;
    if (I < g.Hz && rh < g.eh && j < g.W && c < g.C) {
      const int J = (j + g.pw) / g.sw, rw = (j + g.pw) % g.sw;
      if (J < g.Wz && rw < g.ew)
        v = z[((b * g.Hz + I) * g.Wz + J) * g.ld + static_cast<long long>(rh * g.ew + rw) * g.C + c];
    }
    tile[ty + 8 * k][tx] = v;
  }
  __syncthreads();
  const long long row = (b * g.C * g.H + i) * static_cast<long long>(g.W);
  float r[4] = {0.f, 0.f, 0.f, 0.f};
  if (add != nullptr) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = c0 + ty + 8 * k, j = j0 + tx;
      if (c < g.C && j < g.W) r[k] = __ldg(add + row + static_cast<long long>(c) * g.H * g.W + j);
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = c0 + ty + 8 * k, j = j0 + tx;
    const float v = tile[tx][ty + 8 * k];
    if (c < g.C && j < g.W) x[row + static_cast<long long>(c) * g.H * g.W + j] = add != nullptr ? v + r[k] : v;
  }
}

// y[b, c, p] = act(x[b, p, c] + add[b, c, p]): blocks of 64 pixels x 64 channels.  The addition of a residual and a ReLU
// cost their reads beside the transposition, no pass of their own.
__global__ void __launch_bounds__(256)
nhwc_to_nchw_f32_kernel(const float* __restrict__ x, const float* __restrict__ add, float* __restrict__ y, int C, long long P,
                        long long ld, int relu, int p_tiles, bool quads, const uint8_t* __restrict__ add_mask,
                        uint8_t* __restrict__ mask) {
  __shared__ float tile[64][65];
  const long long b = blockIdx.x / p_tiles, p0 = static_cast<long long>(blockIdx.x % p_tiles) * 64;
  const int c0 = blockIdx.y * 64;
  const bool vec = ld % 4 == 0 && C % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const float* xb = x + b * P * ld;
  if (vec) {
    const int c = (threadIdx.x & 15) * 4, pr = threadIdx.x >> 4;
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long p = p0 + pr + 16 * k;
      v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p < P && c0 + c < C) v[k] = __ldg(reinterpret_cast<const float4*>(xb + p * ld + c0 + c));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      tile[c][pr + 16 * k] = v[k].x;
      tile[c + 1][pr + 16 * k] = v[k].y;
      tile[c + 2][pr + 16 * k] = v[k].z;
      tile[c + 3][pr + 16 * k] = v[k].w;
    }
  } else {
    const int c = threadIdx.x & 63, pr = threadIdx.x >> 6;
    for (int k = 0; k < 16; ++k) {
      const long long p = p0 + pr + 4 * k;
      tile[c][pr + 4 * k] = p < P && c0 + c < C ? xb[p * ld + c0 + c] : 0.f;
    }
  }
  __syncthreads();
  if (quads) {  // channels of whole quads of pixels on 16-byte boundaries
    const int pq = (threadIdx.x & 15) * 4, cq = threadIdx.x >> 4;
    if (p0 + pq >= P) return;
    const long long at = (b * C + c0) * P + p0 + pq;
    float4 r[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = cq + 16 * k;
      r[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (add != nullptr && c0 + c < C) r[k] = __ldg(reinterpret_cast<const float4*>(add + at + c * P));
      if (add_mask != nullptr && c0 + c < C) {
        const uchar4 u = __ldg(reinterpret_cast<const uchar4*>(add_mask + at + c * P));
        r[k] = make_float4(u.x ? r[k].x : 0.f, u.y ? r[k].y : 0.f, u.z ? r[k].z : 0.f, u.w ? r[k].w : 0.f);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = cq + 16 * k;
      if (c0 + c >= C) continue;
      float4 v = make_float4(tile[c][pq], tile[c][pq + 1], tile[c][pq + 2], tile[c][pq + 3]);
      if (add != nullptr) v = make_float4(v.x + r[k].x, v.y + r[k].y, v.z + r[k].z, v.w + r[k].w);
      if (relu) v = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
      *reinterpret_cast<float4*>(y + at + c * P) = v;
      if (mask != nullptr)
        *reinterpret_cast<uchar4*>(mask + at + c * P) = make_uchar4(v.x > 0.f, v.y > 0.f, v.z > 0.f, v.w > 0.f);
    }
    return;
  }
  const int px = threadIdx.x & 63, cr = threadIdx.x >> 6;
  const long long p = p0 + px;
  if (p >= P) return;
  const long long at = (b * C + c0) * P + p;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float r[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int c = cr + 4 * (h * 8 + k);
      r[k] = add != nullptr && c0 + c < C ? __ldg(add + at + c * P) : 0.f;
      if (add_mask != nullptr && c0 + c < C && !__ldg(add_mask + at + c * P)) r[k] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int c = cr + 4 * (h * 8 + k);
      if (c0 + c >= C) continue;
      float v = tile[c][px];
      if (add != nullptr) v += r[k];
      if (relu) v = fmaxf(v, 0.f);
      y[at + c * P] = v;
      if (mask != nullptr) mask[at + c * P] = v > 0.f;
    }
  }
}

bool s2d_ok(int B, const S2d& g) {
  return B > 0 && g.C > 0 && g.H > 0 && g.W > 0 && g.sh > 0 && g.sw > 0 && g.eh > 0 && g.eh <= g.sh && g.ew > 0 &&
         g.ew <= g.sw && g.ph >= 0 && g.pw >= 0 && g.Hz > 0 && g.Wz > 0 &&
         g.ld >= static_cast<long long>(g.eh) * g.ew * g.C && (g.C + 31) / 32 <= 65535;
}
// What the grid of s2d_to_nchw_kernel holds.
bool s2d_grid_ok(int B, const S2d& g) {
  return static_cast<long long>(B) * g.H < 0x7fffffffll && g.W <= 65535 * 32;
}

// Elements of a filter matrix of `rows` rows; 0: no such filter.
long long filter_total(const Filter& f, int rows) {
  if (f.O <= 0 || f.C <= 0 || f.kh <= 0 || f.kw <= 0 || f.sh <= 0 || f.sw <= 0 || f.eh <= 0 || f.ew <= 0) return 0;
  return static_cast<long long>(rows) * f.k2h * f.k2w * f.pitch;
}
// Launches `kernel` for each element, with 32-bit indices where they and a step of the grid beyond them fit.
template <typename K32, typename K64, typename... A>
int for_each_tap(K32 k32, K64 k64, long long total, cudaStream_t stream, A... args) {
  const long long blocks = (total + 255) / 256;
  const int grid = static_cast<int>(blocks < 1184 ? blocks : 1184);
  if (total < 0x7f000000ll)
    k32<<<grid, 256, 0, stream>>>(args..., static_cast<int>(total));
  else
    k64<<<grid, 256, 0, stream>>>(args..., total);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace
}  // namespace fb

// x [B, C, H, W] fp32 -> z [B, Hz, Wz, ld] bf16, every element of it written.  mask (optional): x is the gradient behind
// a ReLU whose result was mask.
namespace {
template <typename M>
int pack_input(const float* x, const M* mask, void* z, int B, int C, int H, int W, int sh, int sw, int eh, int ew, int ph, int pw,
               int Hz, int Wz, long long ld, cudaStream_t stream) {
  fb::S2d g{C, H, W, sh, sw, eh, ew, ph, pw, Hz, Wz, ld};
  const bool plain = sh == 1 && sw == 1 && ph == 0 && pw == 0 && Hz == H && Wz == W;  // images and rows of any size
  if (!fb::s2d_ok(B, g) || (!plain && !fb::s2d_grid_ok(B, g))) return -1;
  if (plain && static_cast<long long>(H) * W < 0x7fffffffll - 64) {  // rows are contiguous: one long row per image
    g.W = g.Wz = H * W;
    g.H = g.Hz = 1;
  }
  const long long q_tiles = (static_cast<long long>(g.Wz) * ew + fb::kTileQ - 1) / fb::kTileQ;
  const long long blocks = q_tiles * B * g.Hz * eh;
  if (blocks > 0x7fffffffll) return -1;
  const dim3 grid(static_cast<unsigned>(blocks), static_cast<unsigned>((C + fb::kTileC - 1) / fb::kTileC));
  // Octets: every pixel's channels start on one.  With a single tap per pixel they may end within one, whose rest is the
  // padding (a forward pass over 32 images of 65 x 30 x 30: 57.7 us channel by channel, 53.0 so).
  const bool vec = ld == static_cast<long long>(eh) * ew * ((C + 7) / 8 * 8) && (C % 8 == 0 || eh * ew == 1) &&
                   reinterpret_cast<uintptr_t>(z) % 16 == 0;
  const bool quads = ew == sw && g.W % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(mask) % (4 * sizeof(M)) == 0;
  const auto kernel = vec ? (quads ? fb::pack_input_kernel<true, true, M> : fb::pack_input_kernel<true, false, M>)
                          : (quads ? fb::pack_input_kernel<false, true, M> : fb::pack_input_kernel<false, false, M>);
  kernel<<<grid, 256, 0, stream>>>(x, mask, static_cast<__nv_bfloat16*>(z), g, static_cast<int>(q_tiles));
  return static_cast<int>(cudaGetLastError());
}
}  // namespace

extern "C" int fb_conv_pack_input(const float* x, const float* mask, void* z, int B, int C, int H, int W, int sh, int sw,
                                  int eh, int ew, int ph, int pw, int Hz, int Wz, long long ld, cudaStream_t stream) {
  return pack_input(x, mask, z, B, C, H, W, sh, sw, eh, ew, ph, pw, Hz, Wz, ld, stream);
}
// The mask as bytes (fb_nhwc_to_nchw_masks); stride 1, no padding.
extern "C" int fb_conv_pack_masked(const float* x, const unsigned char* mask, void* z, int B, int C, int H, int W, long long ld,
                                   cudaStream_t stream) {
  return pack_input<uint8_t>(x, mask, z, B, C, H, W, 1, 1, 1, 1, 0, 0, H, W, ld, stream);
}

// dgrad = 0: out [O, k2h * k2w, pitch], dgrad = 1: out [eh * ew * C, k2h * k2w, pitch] with the taps in reverse order.
extern "C" int fb_conv_pack_filters(const float* w, void* out, int O, int C, int kh, int kw, int sh, int sw, int eh,
                                    int ew, int pitch, int dgrad, cudaStream_t stream) {
  if (sh <= 0 || sw <= 0) return -1;
  const fb::Filter f{O, C, kh, kw, sh, sw, eh, ew, (kh + sh - 1) / sh, (kw + sw - 1) / sw, pitch};
  const int rows = dgrad ? eh * ew * C : O;
  const long long total = fb::filter_total(f, rows);
  if (total <= 0 || pitch < (dgrad ? O : eh * ew * C)) return -1;
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out);
  return dgrad ? fb::for_each_tap(fb::pack_filters_kernel<true, int>, fb::pack_filters_kernel<true, long long>, total,
                                  stream, w, o, f)
               : fb::for_each_tap(fb::pack_filters_kernel<false, int>, fb::pack_filters_kernel<false, long long>, total,
                                  stream, w, o, f);
}

// part [splits, O, k2h * k2w, pitch] -> dw [O, C, kh, kw].
extern "C" int fb_conv_fold_wgrad(const float* part, float* dw, int splits, int O, int C, int kh, int kw, int sh, int sw,
                                  int eh, int ew, int pitch, cudaStream_t stream) {
  if (sh <= 0 || sw <= 0) return -1;
  const fb::Filter f{O, C, kh, kw, sh, sw, eh, ew, (kh + sh - 1) / sh, (kw + sw - 1) / sw, pitch};
  const long long total = fb::filter_total(f, O);
  if (total <= 0 || splits <= 0 || pitch < eh * ew * C) return -1;
  return fb::for_each_tap(fb::fold_wgrad_kernel<int>, fb::fold_wgrad_kernel<long long>, total, stream, part, dw, f, splits);
}

// x[b, c, i, j] = z[b, (i + ph) / sh, (j + pw) / sw, (((i + ph) % sh) * ew + (j + pw) % sw) * C + c], zero where no
// window reaches; plus add (optional, laid out like x).
extern "C" int fb_s2d_nhwc_to_nchw_add(const float* z, const float* add, float* x, int B, int C, int H, int W, int sh, int sw,
                                       int eh, int ew, int ph, int pw, int Hz, int Wz, long long ld, cudaStream_t stream) {
  const fb::S2d g{C, H, W, sh, sw, eh, ew, ph, pw, Hz, Wz, ld};
  if (!fb::s2d_ok(B, g) || !fb::s2d_grid_ok(B, g)) return -1;
  dim3 grid(static_cast<unsigned>(B) * H, static_cast<unsigned>((W + 31) / 32), static_cast<unsigned>((C + 31) / 32));
  fb::s2d_to_nchw_kernel<<<grid, 256, 0, stream>>>(z, add, x, g);
  return static_cast<int>(cudaGetLastError());
}
extern "C" int fb_s2d_nhwc_to_nchw_f32(const float* z, float* x, int B, int C, int H, int W, int sh, int sw, int eh,
                                       int ew, int ph, int pw, int Hz, int Wz, long long ld, cudaStream_t stream) {
  return fb_s2d_nhwc_to_nchw_add(z, nullptr, x, B, C, H, W, sh, sw, eh, ew, ph, pw, Hz, Wz, ld, stream);
}

// y [B, C, P] = x [B, P, ld] (first C channels), plus add [B, C, P] (optional), behind a ReLU with relu = 1.
// add_mask (optional, bytes laid out like add): add counts where it is set; mask (optional): set where y is above zero.
extern "C" int fb_nhwc_to_nchw_masks(const float* x, const float* add, const unsigned char* add_mask, float* y,
                                     unsigned char* mask, int B, int C, long long P, long long ld, int relu, cudaStream_t stream) {
  const long long tiles = (P + 63) / 64;
  if (B <= 0 || C <= 0 || P <= 0 || ld < C || tiles * B > 0x7fffffffll || (C + 63) / 64 > 65535) return -1;
  const dim3 grid(static_cast<unsigned>(tiles * B), static_cast<unsigned>((C + 63) / 64));
  const bool quads = P % 4 == 0 && reinterpret_cast<uintptr_t>(add) % 16 == 0 && reinterpret_cast<uintptr_t>(y) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(add_mask) % 4 == 0 && reinterpret_cast<uintptr_t>(mask) % 4 == 0;
  fb::nhwc_to_nchw_f32_kernel<<<grid, 256, 0, stream>>>(x, add, y, C, P, ld, relu, static_cast<int>(tiles), quads,
                                                       add_mask, mask);
  return static_cast<int>(cudaGetLastError());
}
extern "C" int fb_nhwc_to_nchw_f32(const float* x, const float* add, float* y, int B, int C, long long P, long long ld,
                                   int relu, cudaStream_t stream) {
  return fb_nhwc_to_nchw_masks(x, add, nullptr, y, nullptr, B, C, P, ld, relu, stream);
}
