// dsax_lflag.cu -- the learned RFI flagger: a 4-layer 3x3 conv net
// (8 -> 32 -> 64 -> 64 -> 1 channels, ReLU, 58,337 parameters) over a
// downsampled Stokes-I spectrogram, trained on the plain flagger's masks.
// No reference counterpart: the reference flags only with the statistics
// of src/gpu_flagger.cu, which stay the label source, judge and fallback.
//
// Kernels (NHWC activations, FP32):
//   (features: the plain flagger's staged statistics pass plus
//    lf_stat_features_kernel, both in dsax_flag.cu)
//   lf_labels_kernel   : plain-flagger masks -> pixel labels on the H x C grid
//   conv3x3_kernel     : out = conv(in, w) + b (+ReLU); with flipped and
//                        transposed weights it is also the data gradient,
//                        the ReLU mask of the layer fused into its input load
//   conv3x3_to1_kernel, conv3x3_from1_kernel : the one-channel ends
//   conv3x3_wgrad_kernel, conv3x3_wgrad1_kernel + lf_reduce_kernel : weight /
//                        bias gradients, per-strip partials reduced in a fixed
//                        order
//   lf_bce_kernel      : weighted BCE-with-logits loss and d/dlogits
//   lf_adam_kernel     : Adam update of the FP32 master weights
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "dsax_internal.h"
#include "dsax_lflag.h"

namespace dsax {

__device__ __forceinline__ float slog(float v) { return copysignf(log1pf(fabsf(v)), v); }

// pixel label = chan flag, or (any ts flag in the tds samples and inside the
// guard band)
__global__ void lf_labels_kernel(const uint8_t *chanmask, const uint8_t *tsmask, uint8_t *L,
                                 int B, int T, int C, int tds, int guard) {
  const int H = T / tds;
  const int64_t n = (int64_t)B * H * C;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    const int64_t bh = i / C;
    const int h = (int)(bh % H), b = (int)(bh / H);
    uint8_t v = chanmask[b * C + c];
    if (!v && c >= guard && c < C - guard) {
      const uint8_t *ts = tsmask + (int64_t)b * T + (int64_t)h * tds;
      for (int k = 0; k < tds; ++k) v |= ts[k];
    }
    L[i] = v ? 1 : 0;
  }
}

// ---------------------------------------------------------------- conv3x3
// FP32 convolutions on the FMA pipe (67 TFLOP/s of FMAs at 1.965 GHz), as
// register-tiled products.  A scalar shared load per FMA operand and weights
// read through L1 kept the first form of these kernels at 8.5 TFLOP/s over the
// whole step; with 64 (48 in the weight gradient) accumulators per thread and
// 16-byte shared loads there are 14 to 18 loads to 192 FMAs.
constexpr int kConvRows = 4;     // output rows per CTA

// out[b][y][x][co] = bias[co] + sum_{ky,kx,ci} wt[ky*3+kx][ci][co] *
//                    in'[b][y+ky-1][x+kx-1][ci]     (zero padding)
// in' = in * (gate > 0) when gate != null (ReLU backward of the layer below).
// Thread = 4 consecutive x pixels of one row x 16 output channels.  The rows
// of one ky lie in shared memory by channel [ci][row][x + 1], so that four
// pixels shifted by kx are one or two 16-byte loads; the weights of one tap as
// [ci][co], read as broadcasts.  A sum runs over ky, kx, ci in that order from
// the bias on: another order moves activations near zero across it, and each
// such ReLU shows in the gradients (channels in chunks with all taps of a
// chunk together: 1,450 against 1,690 us for a step of 16 beams x 4,096 x 48,
// but up to 1.7 times the gradients' error against FP64).
template <int CIN, int COUT, bool RELU>
__global__ void __launch_bounds__(256, 2) conv3x3_kernel(const float *__restrict__ in,
                                                         const float *__restrict__ gate,
                                                         const float *__restrict__ wt,
                                                         const float *__restrict__ bias,
                                                         float *__restrict__ out, int B, int H, int W) {
  static_assert(CIN % 4 == 0 && COUT % 16 == 0, "channel tiles");
  constexpr int TH = kConvRows;
  extern __shared__ __align__(16) float csh[];
  const int WP = W + 4, plane = TH * WP;
  float *tile = csh;                              // [CIN][TH][WP]
  float *wsh = csh + CIN * plane;                 // [CIN][COUT]
  const int nrt = (H + TH - 1) / TH;
  const int b = blockIdx.x / nrt, y0 = (blockIdx.x % nrt) * TH;
  const int ngx = W / 4, npg = TH * ngx;          // pixel groups per row, of the CTA
  const int cog = threadIdx.x / npg, rem = threadIdx.x - cog * npg;
  const bool live = cog < COUT / 16;
  const int ty = rem / ngx, x0 = 4 * (rem - ty * ngx);
  float acc[4][16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float bb = bias && live ? bias[cog * 16 + j] : 0.f;
#pragma unroll
    for (int p = 0; p < 4; ++p) acc[p][j] = bb;
  }
#pragma unroll 1
  for (int ky = 0; ky < 3; ++ky) {
#pragma unroll
    for (int kx = 0; kx < 3; ++kx) {
      if (ky || kx) __syncthreads();
      if (kx == 0) {
        for (int i = threadIdx.x; i < (CIN / 4) * plane; i += blockDim.x) {   // (4 channels, pixel)
          const int h = i / plane, pos = i - h * plane;
          const int yy = pos / WP, xx = pos - yy * WP;
          const int gy = y0 + yy + ky - 1, gx = xx - 1;
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          if (gy >= 0 && gy < H && gx >= 0 && gx < W) {
            const int64_t gi = (((int64_t)b * H + gy) * W + gx) * CIN + 4 * h;
            v = *reinterpret_cast<const float4 *>(in + gi);
            if (gate) {
              const float4 g = *reinterpret_cast<const float4 *>(gate + gi);
              v.x = g.x > 0.f ? v.x : 0.f;
              v.y = g.y > 0.f ? v.y : 0.f;
              v.z = g.z > 0.f ? v.z : 0.f;
              v.w = g.w > 0.f ? v.w : 0.f;
            }
          }
          float *t = tile + 4 * h * plane + pos;
          t[0] = v.x;
          t[plane] = v.y;
          t[2 * plane] = v.z;
          t[3 * plane] = v.w;
        }
      }
      const float4 *wg = reinterpret_cast<const float4 *>(wt + (int64_t)(ky * 3 + kx) * CIN * COUT);
      for (int i = threadIdx.x; i < CIN * COUT / 4; i += blockDim.x)
        reinterpret_cast<float4 *>(wsh)[i] = __ldg(wg + i);
      __syncthreads();
      if (!live) continue;
      const float *r = tile + ty * WP + x0;
      const float *wr = wsh + cog * 16;
#pragma unroll 2
      for (int ci = 0; ci < CIN; ++ci) {
        const float4 ra = *reinterpret_cast<const float4 *>(r + ci * plane);
        float v[6] = {ra.x, ra.y, ra.z, ra.w, 0.f, 0.f};
        if (kx) {
          const float2 rb = *reinterpret_cast<const float2 *>(r + ci * plane + 4);
          v[4] = rb.x;
          v[5] = rb.y;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 w = *reinterpret_cast<const float4 *>(wr + ci * COUT + 4 * j);
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            acc[p][4 * j] = fmaf(v[p + kx], w.x, acc[p][4 * j]);
            acc[p][4 * j + 1] = fmaf(v[p + kx], w.y, acc[p][4 * j + 1]);
            acc[p][4 * j + 2] = fmaf(v[p + kx], w.z, acc[p][4 * j + 2]);
            acc[p][4 * j + 3] = fmaf(v[p + kx], w.w, acc[p][4 * j + 3]);
          }
        }
      }
    }
  }
  if (!live || y0 + ty >= H) return;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float4 *o = reinterpret_cast<float4 *>(out + (((int64_t)b * H + y0 + ty) * W + x0 + p) * COUT + cog * 16);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float4 v = make_float4(acc[p][4 * j], acc[p][4 * j + 1], acc[p][4 * j + 2], acc[p][4 * j + 3]);
      if (RELU) {
        v.x = fmaxf(v.x, 0.f);
        v.y = fmaxf(v.y, 0.f);
        v.z = fmaxf(v.z, 0.f);
        v.w = fmaxf(v.w, 0.f);
      }
      o[j] = v;
    }
  }
}

// The last layer, CIN -> 1 (wt[tap][ci]): one warp per output row group of four
// pixels, lanes over the channels (coalesced rows of in), the lanes' partial
// sums by shuffles.  Memory-bound: the activations once, their rows' other
// readers hit L1 / L2.
template <int CIN>
__global__ void __launch_bounds__(256) conv3x3_to1_kernel(const float *__restrict__ in,
                                                          const float *__restrict__ wt,
                                                          const float *__restrict__ bias,
                                                          float *__restrict__ out, int B, int H, int W) {
  static_assert(CIN == 64, "two channels per lane");
  const int lane = threadIdx.x & 31;
  float2 w[9];
#pragma unroll
  for (int t = 0; t < 9; ++t) w[t] = __ldg(reinterpret_cast<const float2 *>(wt + t * CIN) + lane);
  const int ngx = W / 4;
  const int64_t ng = (int64_t)B * H * ngx;
  for (int64_t g = blockIdx.x * (int64_t)(blockDim.x / 32) + threadIdx.x / 32; g < ng;
       g += (int64_t)gridDim.x * (blockDim.x / 32)) {
    const int x0 = 4 * (int)(g % ngx);
    const int64_t row = g / ngx;                  // b * H + y
    const int y = (int)(row % H);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
      if (y + ky - 1 < 0 || y + ky - 1 >= H) continue;
      const float2 *src = reinterpret_cast<const float2 *>(in + ((row + ky - 1) * W) * CIN) + lane;
      float2 v[6];
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        const int x = x0 + i - 1;
        v[i] = x >= 0 && x < W ? __ldg(src + (int64_t)x * (CIN / 2)) : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int kx = 0; kx < 3; ++kx)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          acc[p] = fmaf(v[p + kx].x, w[ky * 3 + kx].x, acc[p]);
          acc[p] = fmaf(v[p + kx].y, w[ky * 3 + kx].y, acc[p]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int p = 0; p < 4; ++p) acc[p] += __shfl_xor_sync(0xffffffffu, acc[p], o);
    if (lane == 0) {
      const float bb = bias[0];
      *reinterpret_cast<float4 *>(out + row * W + x0) =
          make_float4(acc[0] + bb, acc[1] + bb, acc[2] + bb, acc[3] + bb);
    }
  }
}

// Its data gradient, 1 -> COUT (wt[tap][co]): a thread keeps one output
// channel's nine weights and goes along a row; bound by writing out.
template <int COUT>
__global__ void __launch_bounds__(256) conv3x3_from1_kernel(const float *__restrict__ in,
                                                            const float *__restrict__ wt,
                                                            float *__restrict__ out, int B, int H, int W) {
  const int co = threadIdx.x % COUT, xs = threadIdx.x / COUT, nxs = blockDim.x / COUT;
  float w[9];
#pragma unroll
  for (int t = 0; t < 9; ++t) w[t] = __ldg(wt + t * COUT + co);
  for (int64_t row = blockIdx.x; row < (int64_t)B * H; row += gridDim.x) {
    const int y = (int)(row % H);
    for (int x = xs; x < W; x += nxs) {
      float acc = 0.f;
#pragma unroll
      for (int ky = 0; ky < 3; ++ky)
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
          const int yy = y + ky - 1, xx = x + kx - 1;
          const float v = yy >= 0 && yy < H && xx >= 0 && xx < W ? __ldg(in + (row + ky - 1) * W + xx) : 0.f;
          acc = fmaf(v, w[ky * 3 + kx], acc);
        }
      out[(row * W + x) * COUT + co] = acc;
    }
  }
}

// Weight gradient partials over strips of kGradRows rows of one beam:
// part[strip][r][co], r = tap * CIN + ci, and r = 9 CIN the bias: sum over the
// strip's pixels of in[px + tap][ci] * dz'[px][co], dz' = dz * (gate > 0).
// Thread = one ky x three kx x two ci x eight co (co = g + 8 j, so that the
// lanes' rows of dz fall on different banks): 48 sums; for four pixels four
// loads of in and eight of dz, 192 FMAs.
constexpr int kGradRows = 4;     // rows per strip: the length of an FP32 sum
constexpr int kGradTile = 2;     // rows in shared memory at a time
template <int CIN, int CIB, int COUT>
__global__ void __launch_bounds__(3 * (CIB / 2) * (COUT / 8), 2)
    conv3x3_wgrad_kernel(const float *__restrict__ in, const float *__restrict__ dz,
                         const float *__restrict__ gate, float *__restrict__ part, int B, int H, int W) {
  constexpr int kThreads = 3 * (CIB / 2) * (COUT / 8);
  constexpr int RT = kGradTile;
  extern __shared__ __align__(16) float gsh[];
  const int WP = W + 4, plane = (RT + 2) * WP;
  const int S = RT * W + ((RT * W / 4) & 1 ? 0 : 4);   // floats of a dz channel: an odd number of 16 bytes
  float *tile = gsh;                              // [CIB][RT + 2][WP]
  float *dsh = gsh + CIB * plane;                 // [COUT][S]
  const int nst = (H + kGradRows - 1) / kGradRows;
  const int b = blockIdx.x / nst, ys = (blockIdx.x % nst) * kGradRows;
  const int ye = min(H, ys + kGradRows);
  const int c0 = blockIdx.y * CIB;
  const int g = threadIdx.x % (COUT / 8), cp = (threadIdx.x / (COUT / 8)) % (CIB / 2);
  const int ky = threadIdx.x / ((COUT / 8) * (CIB / 2));
  constexpr int kStep = COUT / 8;                 // co = g + kStep j
  const bool with_bias = blockIdx.y == 0 && ky == 1 && cp == 0;
  float acc[2][3][8], accb[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    accb[j] = 0.f;
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int k = 0; k < 3; ++k) acc[c][k][j] = 0.f;
  }
#pragma unroll 1
  for (int y0 = ys; y0 < ye; y0 += RT) {
    if (y0 > ys) __syncthreads();
    constexpr int kQ = CIB / 4;
    for (int i = threadIdx.x; i < kQ * plane; i += kThreads) {
      const int h = i / plane, pos = i - h * plane;
      const int yy = pos / WP, xx = pos - yy * WP;
      const int gy = y0 + yy - 1, gx = xx - 1;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (gy >= 0 && gy < H && gx >= 0 && gx < W)
        v = *reinterpret_cast<const float4 *>(in + (((int64_t)b * H + gy) * W + gx) * CIN + c0 + 4 * h);
      float *t = tile + 4 * h * plane + pos;
      t[0] = v.x;
      t[plane] = v.y;
      t[2 * plane] = v.z;
      t[3 * plane] = v.w;
    }
    for (int i = threadIdx.x; i < (COUT / 4) * RT * W; i += kThreads) {
      const int h = i / (RT * W), px = i - h * RT * W;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (y0 + px / W < ye) {
        const int64_t gi = (((int64_t)b * H + y0) * W + px) * COUT + 4 * h;
        v = *reinterpret_cast<const float4 *>(dz + gi);
        const float4 q = *reinterpret_cast<const float4 *>(gate + gi);
        v.x = q.x > 0.f ? v.x : 0.f;
        v.y = q.y > 0.f ? v.y : 0.f;
        v.z = q.z > 0.f ? v.z : 0.f;
        v.w = q.w > 0.f ? v.w : 0.f;
      }
      float *t = dsh + 4 * h * S + px;
      t[0] = v.x;
      t[S] = v.y;
      t[2 * S] = v.z;
      t[3 * S] = v.w;
    }
    __syncthreads();
#pragma unroll 1
    for (int yy = 0; yy < RT; ++yy) {
      const float *t0 = tile + 2 * cp * plane + (yy + ky) * WP, *t1 = t0 + plane;
      const float *d0 = dsh + g * S + yy * W;
#pragma unroll 1
      for (int x0 = 0; x0 < W; x0 += 4) {
        const float4 a0 = *reinterpret_cast<const float4 *>(t0 + x0);
        const float4 a1 = *reinterpret_cast<const float4 *>(t0 + x0 + 4);
        const float4 b0 = *reinterpret_cast<const float4 *>(t1 + x0);
        const float4 b1 = *reinterpret_cast<const float4 *>(t1 + x0 + 4);
        const float va[6] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y};
        const float vb[6] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 d = *reinterpret_cast<const float4 *>(d0 + kStep * j * S + x0);
          const float dd[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
          for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int kx = 0; kx < 3; ++kx) {
              acc[0][kx][j] = fmaf(va[p + kx], dd[p], acc[0][kx][j]);
              acc[1][kx][j] = fmaf(vb[p + kx], dd[p], acc[1][kx][j]);
            }
          if (with_bias) accb[j] += (dd[0] + dd[1]) + (dd[2] + dd[3]);
        }
      }
    }
  }
  float *o = part + (int64_t)blockIdx.x * (9 * CIN + 1) * COUT;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int co = g + kStep * j;
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int kx = 0; kx < 3; ++kx)
        o[(int64_t)((ky * 3 + kx) * CIN + c0 + 2 * cp + c) * COUT + co] = acc[c][kx][j];
    if (with_bias) o[(int64_t)9 * CIN * COUT + co] = accb[j];
  }
}

// The same for the last layer (64 -> 1, no gate): thread = one ky x three kx of
// one channel, along the rows of a strip of kGradRows1; lanes over the
// channels.  A chain of loads, so short strips (8 rows: 77 us).
constexpr int kGradRows1 = 2;
__global__ void __launch_bounds__(192) conv3x3_wgrad1_kernel(const float *__restrict__ in,
                                                             const float *__restrict__ dz,
                                                             float *__restrict__ part, int B, int H, int W) {
  constexpr int CIN = 64;
  const int nst = (H + kGradRows1 - 1) / kGradRows1;
  const int b = blockIdx.x / nst, ys = (blockIdx.x % nst) * kGradRows1;
  const int ye = min(H, ys + kGradRows1);
  const int ci = threadIdx.x % CIN, ky = threadIdx.x / CIN;
  float acc[3] = {0.f, 0.f, 0.f}, accb = 0.f;
  for (int y = ys; y < ye; ++y) {
    const int gy = y + ky - 1;
    const float *d = dz + ((int64_t)b * H + y) * W;
    const bool in_row = gy >= 0 && gy < H;
    const float *src = in + (((int64_t)b * H + (in_row ? gy : 0)) * W) * CIN + ci;
    float vm = 0.f, v0 = in_row ? __ldg(src) : 0.f;   // in at x - 1, x
#pragma unroll 16
    for (int x = 0; x < W; ++x) {
      const float vp = in_row && x + 1 < W ? __ldg(src + (int64_t)(x + 1) * CIN) : 0.f;
      const float dd = __ldg(d + x);
      acc[0] = fmaf(vm, dd, acc[0]);
      acc[1] = fmaf(v0, dd, acc[1]);
      acc[2] = fmaf(vp, dd, acc[2]);
      accb += dd;
      vm = v0;
      v0 = vp;
    }
  }
  float *o = part + (int64_t)blockIdx.x * (9 * CIN + 1);
#pragma unroll
  for (int kx = 0; kx < 3; ++kx) o[(ky * 3 + kx) * CIN + ci] = acc[kx];
  if (threadIdx.x == 0) o[9 * CIN] = accb;
}

// Sums the strips' partials [nchunk][9*CIN+1][COUT] and writes the gradients in
// the parameter layout W[co][ky][kx][ci], b[co].  Eight threads per output take
// every eighth strip, in FP64, and are added in a fixed order (one thread per
// output and strip after strip: 145 us per layer).
__global__ void __launch_bounds__(256) lf_reduce_kernel(const float *__restrict__ part, int nchunk,
                                                        int cin, int cout, float *gw, float *gb) {
  __shared__ double sh[8][32];
  const int nr = 9 * cin + 1, n = nr * cout;
  const int lane = threadIdx.x & 31, sub = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (i < n) {
#pragma unroll 8
    for (int k = sub; k < nchunk; k += 8) s += (double)__ldg(part + (int64_t)k * n + i);
  }
  sh[sub][lane] = s;
  __syncthreads();
  if (sub || i >= n) return;
  for (int k = 1; k < 8; ++k) s += sh[k][lane];
  const int r = i / cout, co = i - r * cout;
  if (r == 9 * cin) {
    gb[co] = (float)s;
  } else {
    const int tap = r / cin, ci = r - tap * cin;
    gw[((int64_t)co * 9 + tap) * cin + ci] = (float)s;
  }
}

// Every layer's W[co][tap][ci] -> forward layout wt[tap][ci][co] and, for the
// data gradients, wf[8 - tap][co][ci].  Grid (blocks, layers).
struct LfLayoutArgs {
  const float *w[kLfLayers];
  float *wt[kLfLayers], *wf[kLfLayers];
  int cin[kLfLayers], cout[kLfLayers];
};
__global__ void lf_wlayout_kernel(LfLayoutArgs a) {
  const int l = blockIdx.y, cin = a.cin[l], cout = a.cout[l], n = 9 * cin * cout;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int co = i / (9 * cin), tap = (i / cin) % 9, ci = i % cin;
    const float v = a.w[l][i];
    a.wt[l][((int64_t)tap * cin + ci) * cout + co] = v;
    a.wf[l][((int64_t)(8 - tap) * cout + co) * cin + ci] = v;
  }
}

// Weighted BCE-with-logits over valid pixels (guard band excluded), mean;
// writes dlogits and accumulates the loss sum and the valid count.
__global__ void lf_bce_kernel(const float *z, const uint8_t *L, float *dz, double *loss_acc,
                              int B, int H, int W, int guard, float pos_weight, float inv_n) {
  const int64_t n = (int64_t)B * H * W;
  double local = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % W);
    const bool valid = c >= guard && c < W - guard;
    const float zi = z[i], y = L[i] ? 1.f : 0.f;
    const float wgt = valid ? (y > 0.f ? pos_weight : 1.f) : 0.f;
    const float sp = fmaxf(zi, 0.f) + log1pf(expf(-fabsf(zi)));
    local += (double)(wgt * (sp - y * zi));
    const float sig = 1.f / (1.f + expf(-zi));
    dz[i] = wgt * (sig - y) * inv_n;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss_acc, local);
}

__global__ void lf_adam_kernel(float *p, const float *g, float *m, float *v, int n, float lr,
                               float b1, float b2, float eps, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// sigmoid(z) > 0.5  <=>  z > 0; guard band never flagged.
// Pixel mask from the logits; the permanently flagged channels of the
// plain flagger's configuration (inside the guard band) are always set.
__global__ void lf_mask_kernel(const float *z, uint8_t *mask, int64_t n, int W, int guard,
                               float thresh_logit, LfPerm perm) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % W);
    const bool inside = c >= guard && c < W - guard;
    bool pm = false;
    for (int k = 0; k < perm.n; ++k) pm |= perm.ch[k] == c;
    mask[i] = (inside && (z[i] > thresh_logit || pm)) ? 1 : 0;
  }
}

// ---------------------------------------------------------------- launchers
namespace {

template <int CIN, int COUT, bool RELU>
int conv_launch(const float *in, const float *gate, const float *wt, const float *bias, float *out,
                int B, int H, int W, cudaStream_t st) {
  const size_t sh = sizeof(float) * ((size_t)CIN * kConvRows * (W + 4) + CIN * COUT);
  static SmemAttrOnce attr;
  if (smem_attr_once(attr, conv3x3_kernel<CIN, COUT, RELU>, 100 * 1024) != cudaSuccess) return -2;
  const int grid = B * ((H + kConvRows - 1) / kConvRows);
  const int threads = (kConvRows * (W / 4) * (COUT / 16) + 31) / 32 * 32;   // at most 256 (W <= 64)
  conv3x3_kernel<CIN, COUT, RELU><<<grid, threads, sh, st>>>(in, gate, wt, bias, out, B, H, W);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int grad_strips(int B, int H) { return B * ((H + kGradRows - 1) / kGradRows); }

template <int CIN, int CIB, int COUT>
int wgrad_launch(const float *in, const float *dz, const float *gate, float *part, float *gw, float *gb,
                 int B, int H, int W, cudaStream_t st) {
  const size_t sh = sizeof(float) * ((size_t)CIB * (kGradTile + 2) * (W + 4) +
                                     (size_t)COUT * (kGradTile * W + 4));
  static SmemAttrOnce attr;
  if (smem_attr_once(attr, conv3x3_wgrad_kernel<CIN, CIB, COUT>, 100 * 1024) != cudaSuccess) return -2;
  const dim3 grid(grad_strips(B, H), CIN / CIB);
  conv3x3_wgrad_kernel<CIN, CIB, COUT>
      <<<grid, 3 * (CIB / 2) * (COUT / 8), sh, st>>>(in, dz, gate, part, B, H, W);
  lf_reduce_kernel<<<((9 * CIN + 1) * COUT + 31) / 32, 256, 0, st>>>(part, grid.x, CIN, COUT, gw, gb);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace


int lf_labels(const uint8_t *cm, const uint8_t *tm, uint8_t *L, int B, int T, int C, int tds,
              int guard, cudaStream_t st) {
  lf_labels_kernel<<<1024, 256, 0, st>>>(cm, tm, L, B, T, C, tds, guard);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Forward through the 4 layers: acts[0] = features, acts[1..3] post-ReLU,
// acts[4] = logits.  wt[l] are forward-layout weights.
int lf_forward(const LfNet &net, float *const acts[5], int B, int H, int W, cudaStream_t st) {
  int rc = 0;
  rc |= conv_launch<8, 32, true>(acts[0], nullptr, net.wt[0], net.b[0], acts[1], B, H, W, st);
  rc |= conv_launch<32, 64, true>(acts[1], nullptr, net.wt[1], net.b[1], acts[2], B, H, W, st);
  rc |= conv_launch<64, 64, true>(acts[2], nullptr, net.wt[2], net.b[2], acts[3], B, H, W, st);
  conv3x3_to1_kernel<64><<<1184, 256, 0, st>>>(acts[3], net.wt[3], net.b[3], acts[4], B, H, W);
  return rc ? rc : (cudaGetLastError() == cudaSuccess ? 0 : -2);
}

int lf_prepare_weights(const LfNet &net, cudaStream_t st) {
  LfLayoutArgs a;
  for (int l = 0; l < kLfLayers; ++l) {
    a.w[l] = net.w[l];
    a.wt[l] = net.wt[l];
    a.wf[l] = net.wf[l];
    a.cin[l] = kLfCin[l];
    a.cout[l] = kLfCout[l];
  }
  lf_wlayout_kernel<<<dim3(64, kLfLayers), 256, 0, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Backward from dlogits d4 [B][H][W][1]: fills net.gw / net.gb.  The ReLU
// masks are applied as gates (acts[l] > 0) inside the kernels that read the
// gradients.  d_a / d_b: scratch of B*H*W*64 floats each; part: partials.
int lf_backward(const LfNet &net, float *const acts[5], float *d4, float *d_a, float *d_b,
                float *part, int B, int H, int W, cudaStream_t st) {
  int rc = 0;
  // layer 4 (64 -> 1, no ReLU)
  const int n1 = B * ((H + kGradRows1 - 1) / kGradRows1);
  conv3x3_wgrad1_kernel<<<n1, 192, 0, st>>>(acts[3], d4, part, B, H, W);
  lf_reduce_kernel<<<(9 * 64 + 1 + 31) / 32, 256, 0, st>>>(part, n1, 64, 1, net.gw[3], net.gb[3]);
  conv3x3_from1_kernel<64><<<1184, 256, 0, st>>>(d4, net.wf[3], d_a, B, H, W);
  // layer 3 (64 -> 64): dz3 = d_a * (acts[3] > 0)
  rc |= wgrad_launch<64, 16, 64>(acts[2], d_a, acts[3], part, net.gw[2], net.gb[2], B, H, W, st);
  rc |= conv_launch<64, 64, false>(d_a, acts[3], net.wf[2], nullptr, d_b, B, H, W, st);
  // layer 2 (32 -> 64): dz2 = d_b * (acts[2] > 0)
  rc |= wgrad_launch<32, 16, 64>(acts[1], d_b, acts[2], part, net.gw[1], net.gb[1], B, H, W, st);
  rc |= conv_launch<64, 32, false>(d_b, acts[2], net.wf[1], nullptr, d_a, B, H, W, st);
  // layer 1 (8 -> 32): dz1 = d_a * (acts[1] > 0)
  rc |= wgrad_launch<8, 8, 32>(acts[0], d_a, acts[1], part, net.gw[0], net.gb[0], B, H, W, st);
  return rc ? -2 : (cudaGetLastError() == cudaSuccess ? 0 : -2);
}

// (the last layer's shorter strips have one output channel: fewer floats)
size_t lf_part_floats(int B, int H) { return (size_t)grad_strips(B, H) * (9 * 64 + 1) * 64; }

int lf_bce(const float *z, const uint8_t *L, float *dz, double *loss_acc, int B, int H, int W,
           int guard, float pos_weight, float inv_n, cudaStream_t st) {
  lf_bce_kernel<<<512, 256, 0, st>>>(z, L, dz, loss_acc, B, H, W, guard, pos_weight, inv_n);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int lf_adam(LfNet &net, float lr, cudaStream_t st) {
  net.step += 1;
  net.version += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - powf(b1, (float)net.step), c2 = 1.f - powf(b2, (float)net.step);
  lf_adam_kernel<<<128, 256, 0, st>>>(net.params, net.grads, net.m, net.v, lf_nparams(), lr, b1, b2,
                                      1e-8f, c1, c2);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int lf_mask(const float *z, uint8_t *mask, int64_t n, int W, int guard, float thresh_logit,
            const LfPerm &perm, cudaStream_t st) {
  lf_mask_kernel<<<1024, 256, 0, st>>>(z, mask, n, W, guard, thresh_logit, perm);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace dsax
