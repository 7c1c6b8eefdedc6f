// dsax_flag.cu -- the plain RFI flagger on the GPU, statistics and data path.
//
// Replaces src/gpu_flagger.cu, per block in the order of its main loop
// (:1290-1410):
//   scaley (:382-394, once a baseline exists)        -> fused into the
//   calc_spectrum / calc_varspec / calc_maxspec /       statistics pass
//   calc_ppspec (:175-376; the reference calls           (one HBM read)
//   calc_spectrum in calc_maxspec's place at :1334 -- parity mode keeps that)
//   total-power modulation check (:1313-1330)        -> the statistics CTAs
//   channflag x3, simple_channflag (:1340-1347)         (the last one of a
//                                                       beam / of the grid)
//   calc_bpwr (:759-769), gather_mask,               -> flag_apply_kernel
//   flag (:459-474), then make_ts (:414-453),           (reads only the
//   simple_tsflag (:612-653), flagts (:479-494)         flagged chunks; the
//                                                       beam's last CTA does
//                                                       the series tests)
// and fix_zspec (:114-170) + median_calc (:771-798) for the scaley
// baseline.  The shapes the reference hard-codes ([64][16384][1024] uint8,
// ZeroChannels 128, nFiltSize 21, TBIN 128, FBIN 8, T/16) are parameters;
// the filterbank may be uint8 (the reference's type) or FP32.
#include <atomic>
#include <cstdint>
#include <cstring>
#include <type_traits>
#include <cuda.h>
#include <cuda_runtime.h>

#include "dsax_internal.h"
#include "dsax_ptx.cuh"
#include "dsax_scaley.h"
#include "dsax_tmap.h"
#include "../../include/dsax.h"

namespace dsax {

namespace flag {
constexpr int kStatThreads = 256;
constexpr int kTargetCtas = 296;      // statistics CTAs below which time is chunked: two per SM
// Shared memory of a statistics CTA that leaves room for a second one: half of
// an SM's 228 KB, less the 1 KB that each CTA takes and 6.5 KB of static arrays.
constexpr size_t kStatSmem = 114 * 1024 - 1024 - 6656;
constexpr int kMaxChan = 1024;
constexpr int kApplyThreads = 256;    // apply / time-series CTA
constexpr int kApplyRows = 256;       // rows per apply CTA
constexpr int kApplyUnroll = 4;       // row groups of loads in flight
constexpr int kMaxTsBase = 4096;
constexpr int kLfMaxChan = 128;       // learned-flagger features: channels per beam
constexpr int kDecThreads = 256;
}  // namespace flag

// ---------------------------------------------------------------- elements
// Four consecutive channels of one row: FP32 (16 bytes) or uint8 (4 bytes).
template <typename E>
__device__ __forceinline__ void st4(void *p, const float (&v)[4]) {
  if constexpr (std::is_same<E, float>::value) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {   // values are already integers in [0, 255]
    *reinterpret_cast<uint32_t *>(p) = (uint32_t)v[0] | ((uint32_t)v[1] << 8) |
                                       ((uint32_t)v[2] << 16) | ((uint32_t)v[3] << 24);
  }
}
template <typename E>
__device__ __forceinline__ const E *elem_in(const FlagArgs &a) {
  if constexpr (std::is_same<E, float>::value) return a.x; else return a.xu8;
}
template <typename E>
__device__ __forceinline__ E *elem_out(const FlagArgs &a) {
  if constexpr (std::is_same<E, float>::value) return a.xw; else return a.xw8;
}

// scaley (src/gpu_flagger.cu:382-394): (x - spec0) * (SIG / sqrtf(var0)) + MN,
// with the reference's mixed float / double evaluation; uint8 data are
// requantised as (unsigned char)(__float2uint_rn(2 val) / 2), which wraps
// modulo 256 above 255.
template <typename E>
__device__ __forceinline__ float scaley1(float x, float s0, double k, float mn) {
  const float val = (float)((double)(x - s0) * k + (double)mn);
  if constexpr (std::is_same<E, float>::value) {
    return val;
  } else {
    return (float)((__float2uint_rn(2.0f * val) / 2u) & 255u);
  }
}

// The replacement level MN * bpwr as the element type: uint8 is the C
// conversion of `data[idx] = MN * bpwr[bm]` (:473): truncation toward zero,
// clamped to [0, 255] by the device conversion.
template <typename E>
__device__ __forceinline__ E repl_elem(float r) {
  if constexpr (std::is_same<E, float>::value) {
    return r;
  } else {
    return (uint8_t)__float2uint_rz(fminf(r, 255.0f));
  }
}

// The channel decisions of beam b (defined with the order statistics below)
// and the block's total power; both run at the end of the statistics pass.
__device__ void flag_decide_beam(const FlagArgs &a, int b, uint8_t *smem);
__device__ void flag_total_power(const FlagArgs &a);

// ---------------------------------------------------------------- statistics
// One CTA per (channel slab of up to kFlagSlab channels, time chunk, beam).
// A warp takes whole TBIN bins of the chunk (every eighth one), or, where the
// chunk has fewer than eight long ones, an eighth of each.  Its rows come as TMA boxes
// of kBatch passes ([rows][min(nchan, 128) channels], channels past nchan
// zero) into a ring of its own, a.ring - 1 boxes ahead, on its own mbarriers
// (bounded waits, a.wait_limit_ns, recorded in a.err); a pass is as many
// consecutive rows as the lanes hold 4-channel groups of.  So no warp waits
// for another one in the loop.  (Stages for the whole CTA with two block
// barriers and a partly idle row reduction each: 82 against 63 us for
// [256][4096][48] FP32, of which some 26 are what a call costs at any length;
// loads straight into registers: 94.  Scaled uint8 [64][16384][1024]: 1,138
// against 700.)  What bounds it: instructions and waits, not HBM (FP32 [256]
// [4096][48]: DRAM at 40 %, issue slots 50 %).  Scaled uint8 [64][16384][1024]
// reads and writes 2.15 GB at 3.07 TB/s, issue slots 53 %, in 1.73 waves of CTAs
// (a single wave of 256 CTAs: 230 us).
//
// Sums are FP64 for FP32 data and exact integers for uint8: 32 bits within a
// range of rows (a lane's share of a bin or of the tail is at most 49,152 rows
// of an accepted block, so the 255^2 products stay below 2^32; flag_shape_ok),
// 64 bits for the squares from there on, since a lane may have several bins.
// Four rows of uint8 are transposed to words of one channel, whose sum and sum
// of squares are one dp4a each.  A lane's sums are
// combined with the other row phases' in a fixed order, and the chunks' by the
// chunk CTA that finishes last, in chunk order, so results do not depend on
// scheduling.  With a scaley baseline each value is normalised as it is read
// and written back (the statistics then describe the normalised block, as in
// the reference).  Per row the slab's raw sum goes to rowsum (or to ts when
// there is one slab): the lanes' partial sums of a batch of rows meet in the
// warp's own shared buffer.  flag_apply_kernel turns it into the channel-mean
// series after the flagged columns are replaced.
namespace flag {
constexpr int kWarps = kStatThreads / 32;
template <typename E> constexpr int batch() { return std::is_same<E, float>::value ? 8 : 16; }
constexpr int kMaxRing = 4;      // boxes of a warp's ring
constexpr int kPartFields = 5;   // per channel of a chunk: sum, squares, max, bin max, bin min
}  // namespace flag

// kPix: also forms the downsampled spectrogram.  kG: the slab's 4-channel
// groups where they are known when compiling, so that row and table strides are
// constants: 32, a full slab, and 12, the 48 channel groups that the beamformer
// makes of the library's default subband (384 channels).  At 48 channels, us,
// constant / general form (0): masks of 256 x 4,096 FP32 107.6 / 114.7, cleaning
// 64 x 16,384 uint8 113 / 123, learned-flagger features of 256 x 4,096 104 / 124.
// The pixel form has no full slab (it is used up to 64 channels).
template <typename E, bool kPix, int kG>
__global__ void __launch_bounds__(flag::kStatThreads, 2)
    flag_stats_kernel(const __grid_constant__ CUtensorMap tmap, FlagArgs a) {
  constexpr bool kU8 = std::is_same<E, uint8_t>::value;
  constexpr int kBatch = flag::batch<E>();
  constexpr int kWarps = flag::kWarps;
  constexpr bool kRedux = kU8 && kG == 32;     // a warp's pass is one row: warp-wide integer sums
  using Acc = typename std::conditional<kU8, uint32_t, double>::type;   // sums of a lane
  using Vec = typename std::conditional<kU8, uint32_t, float4>::type;   // four channels of a row
  const int slab = (int)blockIdx.x % a.nslab, chunk = (int)blockIdx.x / a.nslab, b = blockIdx.y;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int T = a.ntime, C = a.nchan, TB = a.tbin;
  const int c0 = slab * kFlagSlab;
  const int cs = kG ? 4 * kG : min(kFlagSlab, C - c0);
  const int G4 = kG ? kG : cs >> 2;
  const int bx = kG ? 4 * kG : min(kFlagSlab, C);   // channels of a box row
  const int rpw = 32 / (bx / 4);               // rows of a pass
  // lanes past the last whole row repeat row phase 0 (the same values to the
  // same places); `active` lanes give the totals
  const bool active = lane < rpw * G4;
  const int rp = active ? lane / G4 : 0, g = active ? lane - rp * G4 : lane % G4;
  const bool lead = lane < G4;                 // row phase 0
  const int nbins = T / TB;
  const int bin0 = (int)((int64_t)nbins * chunk / a.nchunk);
  const int bin1 = (int)((int64_t)nbins * (chunk + 1) / a.nchunk);
  E *xw = elem_out<E>(a);
  const bool scale = a.spec0 != nullptr;
  E *const xo = (scale && xw) ? xw + (int64_t)b * T * C + c0 + 4 * g : nullptr;

  extern __shared__ __align__(128) uint8_t fs_raw[];
  __shared__ __align__(8) uint64_t sfull[kWarps][flag::kMaxRing];
  __shared__ volatile int sabort;
  const int GS = G4 | 1;                       // odd row stride of the row buffer
  const int brows = kBatch * rpw;              // rows of a batch
  const int rb = bx * (int)sizeof(E);          // bytes of a staged row
  const int stage_bytes = (brows * rb + 127) & ~127;
  uint8_t *const ring = fs_raw + warp * a.ring * stage_bytes;   // the warp's stages
  uint8_t *const fs_x = fs_raw + kWarps * a.ring * stage_bytes;
  const int rstride = flag_rowbuf(cs, kBatch, rpw, (int)sizeof(Acc));
  Acc *const rbuf = reinterpret_cast<Acc *>(fs_x + warp * rstride);
  double *const sm_part = reinterpret_cast<double *>(fs_x);     // after the loop: [8 rpw][cs]
  // per warp and channel: bin maximum and minimum (bin sums)
  Acc *const sm_bx = reinterpret_cast<Acc *>(fs_x + kWarps * rstride);   // [8][2][cs]
  double *const sm_k = reinterpret_cast<double *>(sm_bx + 2 * kWarps * cs);  // [cs]
  float *const sm_s0 = reinterpret_cast<float *>(sm_k + cs);              // [cs]
  float *const sm_k2 = sm_s0 + cs;                                        // [cs] float(2k)
  uint8_t *const sm_lut = reinterpret_cast<uint8_t *>(sm_k2 + cs);        // uint8: [256][cs]
  const double inv_tb = 1.0 / TB;

  if (scale) {
    for (int c = tid; c < cs; c += flag::kStatThreads) {
      sm_s0[c] = a.spec0[b * C + c0 + c];
      sm_k[c] = (double)a.sig / (double)sqrtf(a.var0[b * C + c0 + c]);
      sm_k2[c] = (float)(2.0 * sm_k[c]);
    }
    __syncthreads();
    if constexpr (kU8) {
      // uint8 has 256 inputs per channel: scaley as a table [x][channel],
      // read by the lanes of a warp (consecutive channel groups) from
      // distinct banks
      for (int i = tid; i < 256 * cs; i += flag::kStatThreads) {
        const int x = i / cs, c = i - x * cs;
        sm_lut[i] = (uint8_t)scaley_u8((float)x, sm_s0[c], sm_k2[c], sm_k[c], a.mn);
      }
    }
  }
  for (int c = lane; c < cs; c += 32) {
    sm_bx[(2 * warp) * cs + c] = kU8 ? (Acc)0 : (Acc)-1e300;
    sm_bx[(2 * warp + 1) * cs + c] = kU8 ? (Acc)0xFFFFFFFFu : (Acc)1e300;
  }
  if (tid == 0) {
    for (int w = 0; w < kWarps; ++w)
      for (int i = 0; i < a.ring; ++i) mbar_init(&sfull[w][i], 1);
    sabort = 0;
    mbar_fence_init();
  }
  __syncthreads();

  using Sq = typename std::conditional<kU8, unsigned long long, double>::type;
  Acc s[4], q[4], bs[4];                       // sums, squares (uint8: of the current range), sums of the current bin
  Sq sq[4];                                    // uint8: squares of the earlier ranges
  float m[4];                                  // maxima (uint8: in mx)
  uint32_t mx[2] = {0u, 0u};                   // uint8 maxima of channels 0, 2 and 1, 3
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    s[j] = 0; q[j] = 0; bs[j] = 0; sq[j] = 0;
    m[j] = -INFINITY;
  }
  // the running pixel of channels lane, lane + 32, ... (sum and maximum over
  // tds rows in row order, FP32), and its rows so far
  constexpr int kPixC = kFlagSlab / 32;
  float px_s[kPixC], px_m[kPixC];
  int px_n = 0;
#pragma unroll
  for (int k = 0; k < kPixC; ++k) {
    px_s[k] = 0.0f;
    px_m[k] = -INFINITY;
  }

  // scaley of four channels by the table (one extraction, one multiply-add
  // and one load per sample: explicit shared addresses keep it at that)
  const uint32_t lut_base = smem_u32(sm_lut) + 4u * g;
  auto lut4 = [&](uint32_t w) -> uint32_t {
    uint32_t y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      asm("ld.shared.u8 %0, [%1];" : "=r"(y[j]) : "r"(__byte_perm(w, 0u, 0x4440u + j) * cs + lut_base + j));
    return __byte_perm(__byte_perm(y[0], y[1], 0x0040u), __byte_perm(y[2], y[3], 0x0040u), 0x5410u);
  };
  auto take_u8 = [&](const uint32_t (&w)[4]) {
    const uint32_t t0 = __byte_perm(w[0], w[1], 0x5140u), t1 = __byte_perm(w[0], w[1], 0x7362u);
    const uint32_t t2 = __byte_perm(w[2], w[3], 0x5140u), t3 = __byte_perm(w[2], w[3], 0x7362u);
    const uint32_t x[4] = {__byte_perm(t0, t2, 0x5410u), __byte_perm(t0, t2, 0x7632u),
                           __byte_perm(t1, t3, 0x5410u), __byte_perm(t1, t3, 0x7632u)};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      bs[j] = (Acc)__dp4a(x[j], 0x01010101u, (uint32_t)bs[j]);
      q[j] = (Acc)__dp4a(x[j], x[j], (uint32_t)q[j]);
    }
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
      mx[0] = __vimax3_u16x2(mx[0], w[k] & 0x00FF00FFu, w[k + 1] & 0x00FF00FFu);
      mx[1] = __vimax3_u16x2(mx[1], (w[k] >> 8) & 0x00FF00FFu, (w[k + 1] >> 8) & 0x00FF00FFu);
    }
  };
  auto put_row = [&](int t, double r) {
    if (a.nslab == 1)
      a.ts[(int64_t)b * T + t] = a.ts_mean ? (float)(r / C) : (float)r;
    else
      a.rowsum[((int64_t)b * a.nslab + slab) * T + t] = (float)r;
  };
  // one batch of rows from t on, the first `n` of them (kWhole: all brows)
  auto batch = [&](auto whole_t, const uint8_t *sp, int t, int n) {
    constexpr bool kWhole = decltype(whole_t)::value;
    const uint32_t src = smem_u32(sp) + rp * rb + g * (int)sizeof(Vec);
    [[maybe_unused]] Acc *const rs = rbuf + rp * GS + g;
    // (uint8: at most 2^28 samples of a beam, so 32-bit offsets)
    using Off = typename std::conditional<kU8, uint32_t, int64_t>::type;
    E *const dst = xo;
    const Off doff = (Off)(t + rp) * (Off)C, step = (Off)rpw * (Off)C;
    [[maybe_unused]] uint32_t rsum[kBatch / 2];   // full uint8 slabs: row sums of two rows each
    if constexpr (kU8) {
#pragma unroll
      for (int u = 0; u < kBatch; u += 4) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[i]) : "r"(src + (u + i) * rpw * rb));
        if (scale) {
#pragma unroll
          for (int i = 0; i < 4; ++i) w[i] = lut4(w[i]);
        }
        if constexpr (!kWhole) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (rp + (u + i) * rpw >= n) w[i] = 0u;
        }
        if (dst) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (kWhole || rp + (u + i) * rpw < n)
              __stcs(reinterpret_cast<uint32_t *>(dst + (doff + (u + i) * step)), w[i]);
        }
        if constexpr (kRedux) {   // a row of at most 128 x 255 fits 16 bits
#pragma unroll
          for (int i = 0; i < 4; i += 2)
            rsum[(u + i) / 2] = __reduce_add_sync(
                0xffffffffu, __dp4a(w[i], 0x01010101u, 0u) + (__dp4a(w[i + 1], 0x01010101u, 0u) << 16));
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) rs[(u + i) * rpw * GS] = __dp4a(w[i], 0x01010101u, 0u);
        }
        take_u8(w);
      }
    } else {
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        if (kWhole || rp + u * rpw < n) {
          float x[4];
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                       : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(src + u * rpw * rb));
          if (scale) {
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = scaley1<E>(x[j], sm_s0[4 * g + j], sm_k[4 * g + j], a.mn);
            if (dst) st4<E>(dst + (doff + u * step), x);
          }
          const double d0 = (double)x[0], d1 = (double)x[1], d2 = (double)x[2], d3 = (double)x[3];
          bs[0] += d0; bs[1] += d1; bs[2] += d2; bs[3] += d3;
          q[0] += d0 * d0; q[1] += d1 * d1; q[2] += d2 * d2; q[3] += d3 * d3;
#pragma unroll
          for (int j = 0; j < 4; ++j) m[j] = fmaxf(m[j], x[j]);
          rs[u * rpw * GS] = ((d0 + d1) + d2) + d3;
        }
      }
    }
    if constexpr (kPix) {   // from the staged rows (whole pixels per range of rows)
      const float *sf = reinterpret_cast<const float *>(sp);
      const int nr = kWhole ? brows : n;
#pragma unroll 1
      for (int r0 = 0; r0 < nr;) {
        const int r1 = min(nr, r0 + a.tds - px_n);
        px_n += r1 - r0;
#pragma unroll 4
        for (int r = r0; r < r1; ++r)
#pragma unroll
          for (int k = 0; k < kPixC; ++k)
            if (lane + 32 * k < cs) {
              const float v = sf[r * bx + lane + 32 * k];
              px_s[k] += v;
              px_m[k] = fmaxf(px_m[k], v);
            }
        r0 = r1;
        if (px_n < a.tds) break;
        px_n = 0;
        const int64_t o = ((int64_t)b * (T / a.tds) + (t + r1) / a.tds - 1) * C + c0;
#pragma unroll
        for (int k = 0; k < kPixC; ++k)
          if (lane + 32 * k < cs) {
            a.pix_sum[o + lane + 32 * k] = px_s[k];
            a.pix_max[o + lane + 32 * k] = px_m[k];
            px_s[k] = 0.0f;
            px_m[k] = -INFINITY;
          }
      }
    }
    if constexpr (kRedux) {   // lane k keeps and writes the sum of row k
      uint32_t v = 0u;
#pragma unroll
      for (int k = 0; k < kBatch / 2; ++k)
        if ((lane >> 1) == k) v = rsum[k];
      if (lane < (kWhole ? kBatch : n)) put_row(t + lane, (double)((lane & 1) ? v >> 16 : v & 0xFFFFu));
      return;
    }
    __syncwarp();
    // row sums: lr lanes per row, then a shuffle tree (batches of 8 or 16 rows
    // fill the warp exactly; larger ones take one lane per row)
    static_assert(kBatch == 8 || kBatch == 16, "every lane takes part in the row shuffles");
    const int lr = brows <= 8 ? 4 : brows <= 16 ? 2 : 1;
    const int sub = lane & (lr - 1);
    for (int k = lane / lr; k < brows; k += 32 / lr) {
      const Acc *w = rbuf + k * GS;
      Acc a0 = 0, a1 = 0;
      int e = sub;
      for (; e + lr < G4; e += 2 * lr) {
        a0 += w[e];
        a1 += w[e + lr];
      }
      if (e < G4) a0 += w[e];
      a0 += a1;
      for (int o = 1; o < lr; o <<= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, o);
      if (sub == 0 && (kWhole || k < n)) put_row(t + k, (double)a0);
    }
    __syncwarp();
  };
  // `count` ranges of n rows, tstep apart from t0 on: boxes of brows rows (the
  // last of a range may reach past it), a.ring - 1 ahead through all of the
  // ranges, taken one after the other; `end` after each range
  uint32_t is = 0, cs_i = 0, cs_ph = 0;        // ring positions: issue, consume (and its parity)
  auto run = [&](int t0, int n, int tstep, int count, auto end) {
    int ir = 0, ik = 0;                        // next box to issue
    auto issue = [&]() {
      if (ir >= count || n <= 0) return;
      if (lane == 0) {
        mbar_arrive_expect_tx(&sfull[warp][is], (uint32_t)(brows * rb));
        tma_load_2d(smem_u32(ring) + is * stage_bytes, &tmap, c0, b * T + t0 + ir * tstep + ik,
                    &sfull[warp][is]);
      }
      if (++is == (uint32_t)a.ring) is = 0;
      ik += brows;
      if (ik >= n) {
        ik = 0;
        ++ir;
      }
    };
    for (int i = 0; i + 1 < a.ring; ++i) issue();
#pragma unroll 1
    for (int r = 0; r < count; ++r) {
#pragma unroll 1
      for (int k0 = 0; k0 < n; k0 += brows) {
        issue();
        const bool ok = mbar_wait_bounded(&sfull[warp][cs_i], cs_ph, &sabort, a.err, DEV_ERR_WAIT_FULL,
                                          a.wait_limit_ns);
        if (!__all_sync(0xffffffffu, ok)) {    // recorded in a.err; the box lands before the CTA exits
          volatile int no_abort = 0;
          mbar_wait_bounded(&sfull[warp][cs_i], cs_ph, &no_abort, a.err, DEV_ERR_WAIT_FULL,
                            drain_limit(a.wait_limit_ns));
        } else {
          const uint8_t *sp = ring + cs_i * stage_bytes;
          const int t = t0 + r * tstep + k0;
          if (k0 + brows <= n) batch(std::true_type{}, sp, t, brows);
          else batch(std::false_type{}, sp, t, n - k0);
        }
        // the stage's reads before the box that overwrites it
        fence_proxy_async_smem();
        __syncwarp();
        if (++cs_i == (uint32_t)a.ring) {
          cs_i = 0;
          cs_ph ^= 1u;
        }
      }
      end();
    }
  };
  // the bin's sums over the row phases -> its extremes (phase 0's lanes)
  auto bin_total = [&](int j) -> Acc {
    Acc t = bs[j];
    for (int k = 1; k < rpw; ++k) t += __shfl_sync(0xffffffffu, bs[j], (lane + k * G4) & 31);
    return t;
  };
  // Segments: all of the warp's whole bins in one, or, with fewer bins than
  // warps, one per bin (an eighth of its rows, in passes or pixel rows, per
  // warp; the bin's sums combined by the CTA); then the rows beyond the last
  // whole bin: everything but the bins.  (One loop, so that the row code exists
  // once.)
  // (Split bins go one after the other, each with its latency and barriers
  // however short; a warp per bin leaves warps idle.  Up to 2^n boxes in each of
  // n bins the warp is no slower.  256 beams, us, warp / split: 64 channels, one
  // bin of 4 boxes 35.8 / 31.9, 256 channels, two of 8 81 / 68, three of 16 130 /
  // 116; 64 channels, four of 8 48.4 / 48.3, seven of 8 60 / 64.)
  const bool by_warp = bin1 - bin0 >= kWarps || (TB + brows - 1) / brows <= 1 << (bin1 - bin0);
  const int nbseg = by_warp ? 1 : bin1 - bin0;
  const int ntail = chunk == a.nchunk - 1 ? T - nbins * TB : 0;
  // a short tail goes to a warp that has no bin
  const bool tail_in = by_warp && bin1 - bin0 < kWarps && ntail > 0 && ntail <= 2 * brows;
  const int nseg = nbseg + (ntail > 0 && !tail_in ? 1 : 0);
#pragma unroll 1
  for (int seg = 0; seg < nseg; ++seg) {
    const bool tail = seg == nbseg, whole = by_warp && !tail;
    int t0 = (bin0 + warp) * TB, n = TB, count = (bin1 - bin0 - warp + kWarps - 1) / kWarps;
    const bool my_tail = whole && tail_in && warp == bin1 - bin0;
    if (my_tail) {
      t0 = nbins * TB;
      n = ntail;
      count = 1;
    }
    if (!whole) {
      const int s0 = tail ? nbins * TB : (bin0 + seg) * TB, len = tail ? T - s0 : TB;
      const int unit = kPix ? a.tds : rpw;
      const int per = ((len + unit - 1) / unit + kWarps - 1) / kWarps * unit;
      const int r0 = min(len, warp * per), r1 = min(len, (warp + 1) * per);
      t0 = s0 + r0;
      n = r1 - r0;
      count = 1;
    }
    run(t0, n, kWarps * TB, count, [&]() {
      if constexpr (kU8) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          sq[j] += q[j];
          q[j] = 0;
        }
      }
      if (whole) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const Acc t = bin_total(j);
          if (lead && !my_tail) {
            Acc *e = sm_bx + 2 * warp * cs + 4 * g + j;
            e[0] = max(e[0], t);
            e[cs] = min(e[cs], t);
          }
          s[j] += bs[j];
          bs[j] = 0;
        }
      }
    });
    if (whole) continue;
    Acc *const bp = reinterpret_cast<Acc *>(fs_x);
    if (!tail) __syncthreads();   // the row buffers become [8][cs] partial bin sums
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const Acc t = bin_total(j);
      if (lead && !tail) bp[warp * cs + 4 * g + j] = t;
      s[j] += bs[j];
      bs[j] = 0;
    }
    if (tail) continue;
    __syncthreads();
    for (int c = tid; c < cs; c += flag::kStatThreads) {
      Acc t = 0;
      for (int w = 0; w < kWarps; ++w) t += bp[w * cs + c];
      sm_bx[c] = max(sm_bx[c], t);
      sm_bx[cs + c] = min(sm_bx[cs + c], t);
    }
    __syncthreads();
  }
  __syncthreads();
  if (sabort) return;   // recorded in a.err; no statistics from this CTA
  // per-channel totals over the row phases of every warp, in order
  const int P = kWarps * rpw;
  double tot[3] = {0.0, 0.0, -INFINITY};
#pragma unroll
  for (int pass = 0; pass < 3; ++pass) {
    __syncthreads();
    if (active) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double mj = kU8 ? (double)((mx[j & 1] >> (8 * (j & 2))) & 0xFFFFu) : (double)m[j];
        sm_part[(warp * rpw + rp) * cs + 4 * g + j] = pass == 0 ? (double)s[j] : pass == 1 ? (double)(kU8 ? sq[j] : (Sq)q[j]) : mj;
      }
    }
    __syncthreads();
    if (tid < cs) {
      if (pass < 2) {
        double a0 = 0.0, a1 = 0.0;
        for (int k = 0; k + 1 < P; k += 2) {
          a0 += sm_part[k * cs + tid];
          a1 += sm_part[(k + 1) * cs + tid];
        }
        tot[pass] = a0 + a1;                   // (P is a multiple of 8)
      } else {
        for (int k = 0; k < P; ++k) tot[2] = fmax(tot[2], sm_part[k * cs + tid]);
      }
    }
  }
  double bmax = -1e300, bmin = 1e300;          // bin sums
  if (tid < cs && bin1 > bin0) {
    Acc hi = sm_bx[tid], lo = sm_bx[cs + tid];
    for (int w = 1; w < kWarps; ++w) {
      hi = max(hi, sm_bx[2 * w * cs + tid]);
      lo = min(lo, sm_bx[(2 * w + 1) * cs + tid]);
    }
    bmax = (double)hi;
    bmin = (double)lo;
  }
  __shared__ int last_sh;
  if (a.nchunk > 1) {
    // the chunk's partial results; the (beam, slab)'s last chunk CTA combines
    // them in chunk order (nothing waits)
    double *const part = a.part + ((int64_t)b * a.nslab + slab) * a.nchunk * flag::kPartFields * kFlagSlab;
    if (tid < cs) {
      double *o = part + (int64_t)chunk * flag::kPartFields * kFlagSlab + tid;
      o[0] = tot[0];
      o[kFlagSlab] = tot[1];
      o[2 * kFlagSlab] = tot[2];
      o[3 * kFlagSlab] = bmax;
      o[4 * kFlagSlab] = bmin;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0)
      last_sh = atomicAdd(a.ctr + flag_ctr_chunk(a.nbeam) + b * a.nslab + slab, 1) == a.nchunk - 1;
    __syncthreads();
    if (!last_sh) {
      if (!a.decide || (!a.modcheck && !a.tpwr_out)) return;
    } else {
      __threadfence();
      if (tid < cs) {
        tot[0] = tot[1] = 0.0;
        tot[2] = -INFINITY;
        bmax = -1e300;
        bmin = 1e300;
        for (int k = 0; k < a.nchunk; ++k) {
          const double *o = part + (int64_t)k * flag::kPartFields * kFlagSlab + tid;
          tot[0] += __ldcg(o);
          tot[1] += __ldcg(o + kFlagSlab);
          tot[2] = fmax(tot[2], __ldcg(o + 2 * kFlagSlab));
          bmax = fmax(bmax, __ldcg(o + 3 * kFlagSlab));
          bmin = fmin(bmin, __ldcg(o + 4 * kFlagSlab));
        }
      }
    }
  }
  const bool owner = a.nchunk == 1 || last_sh;
  if (owner && tid < cs) {
    const double mean = tot[0] / T;
    const double var = fmax(tot[1] / T - mean * mean, 0.0);
    const int o = b * C + c0 + tid;
    a.spec[o] = (float)mean;
    a.var[o] = (float)var;
    a.maxs[o] = a.parity ? (float)mean : (float)tot[2];
    // (both products rounded: fused into one the difference of equal bins is not 0)
    a.pp[o] = nbins > 0 ? (float)(__dmul_rn(bmax, inv_tb) - __dmul_rn(bmin, inv_tb)) : 0.0f;
  }
  if (!a.decide) return;
  // The last slab CTA of the beam makes its channel decisions, and the last
  // CTA of the grid the block-level total power: each CTA publishes its
  // statistics (fence) before counting itself in; nothing waits.
  __threadfence();
  __syncthreads();
  if (owner) {
    if (tid == 0) last_sh = a.nslab == 1 ? 1 : (atomicAdd(a.ctr + b, 1) == a.nslab - 1);
    __syncthreads();
    if (last_sh) {
      __threadfence();
      flag_decide_beam(a, b, fs_raw);
    }
  }
  if (!a.modcheck && !a.tpwr_out) return;
  __syncthreads();
  if (tid == 0) last_sh = atomicAdd(a.ctr + 2 * a.nbeam, 1) == (int)(gridDim.x * gridDim.y) - 1;
  __syncthreads();
  if (last_sh) {
    __threadfence();
    flag_total_power(a);
  }
}

// ---------------------------------------------------------------- decisions
// (the order-statistic helpers: radix select below, the rank-count medians
// and the learned-flagger feature kernel)
// The k-th smallest of v[0..n) (0-based; the value rank counting with
// ties by index returns) by a four-pass MSB-first radix select over
// order-preserving 32-bit keys: per pass a 256-bin shared histogram of the
// candidates that still match the selected prefix, then one warp finds the
// bin holding rank k.  O(n) work instead of O(n^2); finite inputs.
__device__ __forceinline__ uint32_t ordered_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// Few values are ranked by counting instead (two barriers for 16), one a thread:
// a second one doubles the loop.  A call of 256 beams x 64 samples, us, counting /
// select by 64 threads: 16 channels 28 / 36, 48 32 / 38, 64 36 / 41, 72 37 / 34, 96
// 40 / 37, 128 46 / 36; of 4,096 samples x 8 channels with 96 in the time series'
// base, by 256 threads, 16 beams 35.0 / 36.2, 256 beams 69.1 / 68.7, with 128 36.0 /
// 36.2 and 71.5 / 68.7.
constexpr int kRankMax = 96;
__device__ __forceinline__ float grp_radix_select(const float *v, int n, int k, uint32_t *hist,
                                                  uint32_t *sel, int gtid, int gsize, int bid) {
  if (n <= gsize && n <= kRankMax) {
    if (gtid < n) {
      const uint32_t x = ordered_key(v[gtid]);
      int r = 0;
#pragma unroll 4
      for (int q = 0; q < n; ++q) {
        const uint32_t y = ordered_key(v[q]);
        r += y < x || (y == x && q < gtid);
      }
      if (r == k) sel[0] = __float_as_uint(v[gtid]);
    }
    named_bar(bid, gsize);
    const float out = __uint_as_float(sel[0]);
    named_bar(bid, gsize);
    return out;
  }
  uint32_t prefix = 0u, pmask = 0u;
  int kk = k;
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int i = gtid; i < 256; i += gsize) hist[i] = 0u;
    named_bar(bid, gsize);
    for (int i = gtid; i < n; i += gsize) {
      const uint32_t u = ordered_key(v[i]);
      if ((u & pmask) == prefix) atomicAdd(&hist[(u >> shift) & 255u], 1u);
    }
    named_bar(bid, gsize);
    if (gtid < 32) {   // the first warp: bin holding rank kk
      uint32_t c[8], tot = 0u;
#pragma unroll
      for (int e = 0; e < 8; ++e) { c[e] = hist[8 * gtid + e]; tot += c[e]; }
      uint32_t incl = tot;   // inclusive scan over lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (gtid >= o) incl += y;
      }
      const uint32_t excl = incl - tot;
      if (excl <= (uint32_t)kk && (uint32_t)kk < incl) {
        uint32_t run = excl;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if ((uint32_t)kk < run + c[e]) {
            sel[0] = (uint32_t)(8 * gtid + e);
            sel[1] = (uint32_t)kk - run;
            break;
          }
          run += c[e];
        }
      }
    }
    named_bar(bid, gsize);
    prefix |= sel[0] << shift;
    pmask |= 0xFFu << shift;
    kk = (int)sel[1];
    named_bar(bid, gsize);
  }
  const uint32_t u = (prefix & 0x80000000u) ? (prefix & 0x7FFFFFFFu) : ~prefix;
  return __uint_as_float(u);
}

// The same as a call, for the channel decisions: a CTA runs them once, and what
// they cost is mostly fetching their instructions.
__device__ __noinline__ float grp_select_call(const float *v, int n, int k, uint32_t *hist,
                                              uint32_t *sel, int gtid, int gsize, int bid) {
  return grp_radix_select(v, n, k, hist, sel, gtid, gsize, bid);
}

// One window of channflag's detrend: v - lower median of x[0..kF), the median
// by rank counting with ties by index, in registers (a thread per window;
// with a thread per window element and shared loads it was 70 us of the 1,024
// channels' decisions).  Nothing is written where no element has the rank: the
// window is mostly NaN, and its caller's NaN stays, which no test flags.
template <int kF>
__device__ __forceinline__ void window_median(const float *x, float v, float *out) {
  float e[kF];
  int r[kF];
#pragma unroll
  for (int i = 0; i < kF; ++i) {
    e[i] = x[i];
    r[i] = 0;
  }
#pragma unroll
  for (int i = 0; i < kF; ++i)
#pragma unroll
    for (int q = i + 1; q < kF; ++q) {
      r[i] += e[q] < e[i];
      r[q] += e[i] <= e[q];
    }
#pragma unroll
  for (int i = 0; i < kF; ++i)
    if (r[i] == (kF + 1) / 2 - 1) *out = v - e[i];
}

// The windows of channflag (src/gpu_flagger.cu:655-720) of the three spectra at
// sb0, sb0 + 3 C and sb0 + 6 C, each detrended into its next C floats: forward
// nFiltSize-channel median detrend inside the guard band, by `gsize` threads.
__device__ void grp_detrend3(float *sb0, const FlagArgs &a, int gtid, int gsize) {
  const int C = a.nchan, G = a.guard, F = a.filt, n = C - 2 * G;
  const int kf = (F + 1) / 2 - 1;
  if (F == 21 && n > 128) {   // nFiltSize; few channels: not worth the unrolled code
    for (int id = gtid; id < 3 * n; id += gsize) {
      const int k = id / n, jj = id - k * n;
      float *sb = sb0 + 3 * C * k;
      const int j = G + jj, w0 = (C - G - j >= F) ? j : C - G - F;
      window_median<21>(sb + w0, sb[j], sb + C + jj);
    }
    return;
  }
  for (int id = gtid; id < 3 * n * F; id += gsize) {
    const int k = id / (n * F), idx = id - k * n * F;
    const float *sb = sb0 + 3 * C * k;
    float *corr = sb0 + 3 * C * k + C;
    const int jj = idx / F, i = idx - jj * F;
    const int j = G + jj;
    const int w0 = (C - G - j >= F) ? j : C - G - F;
    const float x = sb[w0 + i];
    int r = 0;
    for (int q = 0; q < F; ++q) {
      const float y = sb[w0 + q];
      r += (y < x) || (y == x && q < i);
    }
    if (r == kf) corr[jj] = sb[j] - x;
  }
}

// channflag's decisions from the detrended spectrum: |x| > Thr * MAD inside
// the guard band (compared against 0, as the reference does).  Medians are
// lower medians (medval, :534-556).
__device__ void grp_channflag(float thr, const FlagArgs &a, uint8_t *mask, const float *corr,
                              float *tmp, uint32_t *hist, uint32_t *sel, int gtid, int gsize,
                              int bid) {
  const int C = a.nchan, G = a.guard, n = C - 2 * G;
  const int k = (n + 1) / 2 - 1;
  const float med = grp_select_call(corr, n, k, hist, sel, gtid, gsize, bid);
  for (int i = gtid; i < n; i += gsize) tmp[i] = fabsf(corr[i] - med);
  named_bar(bid, gsize);
  const float mad = grp_select_call(tmp, n, k, hist, sel, gtid, gsize, bid);
  for (int i = gtid; i < n; i += gsize) {
    const float v = corr[i];
    if (v > thr * mad || v < -thr * mad) mask[G + i] = 1;
  }
}

// The channel decisions of beam b, by the 256 threads of the statistics CTA
// that completed the beam: the four tests concurrently in four groups of 64
// threads -- channflag(spec - oldspec, Thr), channflag(var, Thr + 0.5),
// channflag(max, Thr), simple_channflag(pp, Thr / sqrt(FBIN)) (one-sided
// FBIN-channel mean; parity mode keeps the reference's spec[j] sum, :594) --
// ORed into one mask, plus the permanent flag channels
// (src/gpu_flagger.cu:1340-1347).  smem: 12 nchan floats + nchan bytes.
__device__ void flag_decide_beam(const FlagArgs &a, int b, uint8_t *smem) {
  const int tid = threadIdx.x, warp = tid >> 5;
  const int C = a.nchan, G = a.guard, n = C - 2 * G;
  float *dsh = reinterpret_cast<float *>(smem);                 // [4 groups][3][C]
  uint8_t *cmask = reinterpret_cast<uint8_t *>(dsh + 12 * C);   // [C]
  __shared__ uint32_t hist[4][256], sel[4][2];
  for (int c = tid; c < C; c += flag::kStatThreads) cmask[c] = 0;
  __syncthreads();
  const int g = warp >> 1, gsize = 64, gtid = tid - 64 * g, bid = 1 + g;
  float *sb = dsh + g * 3 * C, *corr = sb + C, *tm = corr + C;
  const float *src = g == 0 ? a.spec : g == 1 ? a.var : g == 2 ? a.maxs : a.pp;
  for (int c = gtid; c < C; c += gsize) {
    sb[c] = src[b * C + c] - ((g == 0 && a.oldspec) ? a.oldspec[b * C + c] : 0.0f);
    corr[c] = NAN;   // what a window without a median leaves
  }
  __syncthreads();
  // the three detrends by the whole CTA, then a test per group
  grp_detrend3(dsh, a, tid, flag::kStatThreads);
  __syncthreads();
  if (g < 3) {
    const float thr = g == 1 ? a.thresh + a.var_add : a.thresh;
    grp_channflag(thr, a, cmask, corr, tm, hist[g], sel[g], gtid, gsize, bid);
  } else {   // simple_channflag (:559-610)
    for (int i = gtid; i < n; i += gsize) corr[i] = sb[G + i];
    named_bar(bid, gsize);
    const int k = (n + 1) / 2 - 1;
    const float med = grp_select_call(corr, n, k, hist[g], sel[g], gtid, gsize, bid);
    for (int i = gtid; i < n; i += gsize) tm[i] = fabsf(corr[i] - med);
    named_bar(bid, gsize);
    const float mad = grp_select_call(tm, n, k, hist[g], sel[g], gtid, gsize, bid);
    const float mythr = (float)((double)a.thresh / sqrt((double)a.fbin));
    for (int j = G + gtid; j < C - G - a.fbin; j += gsize) {
      float vv = 0.0f;
      for (int q = 0; q < a.fbin; ++q) vv += a.parity ? sb[j] : sb[j + q];
      vv = vv / (float)a.fbin - med;
      if (vv > mythr * mad) cmask[j] = 1;
    }
  }
  __syncthreads();
  if (tid == 0)
    for (int q = 0; q < a.nperm; ++q) {
      const int j = a.perm[q];
      if (j >= G && j < C - G) cmask[j] = 1;
    }
  __syncthreads();
  int nflag = 0;
  for (int c = tid; c < C; c += flag::kStatThreads) {
    a.chanmask[b * C + c] = cmask[c];
    nflag += cmask[c];
  }
  if (nflag && a.counts) atomicAdd(a.counts, nflag);
}

// Total power of the block (every beam's spectrum summed in FP64 in a fixed
// order) and, with modcheck, the modulation test against the previous
// flagged block (:1313-1330): at or above mod_thresh the block is replaced
// by the noise block and nothing is flagged.  One CTA, the last one of the
// statistics grid.
__device__ void flag_total_power(const FlagArgs &a) {
  __shared__ double red[flag::kStatThreads];
  const int tid = threadIdx.x, BC = a.nbeam * a.nchan;
  double acc = 0.0;
  // (in order; the loads of 16 values are in flight together)
  for (int i0 = tid; i0 < BC; i0 += 16 * flag::kStatThreads) {
    float v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int i = i0 + k * flag::kStatThreads;
      v[k] = i < BC ? __ldcg(a.spec + i) : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (i0 + k * flag::kStatThreads < BC) acc += v[k];
  }
  red[tid] = acc;
  __syncthreads();
  if (tid == 0) {
    double tp = 0.0;
    for (int k = 0; k < flag::kStatThreads; ++k) tp += red[k];
    int rep = 0;
    if (a.modcheck) {
      const double prev = *a.prev_tpwr;
      if (prev > 0.0 && fabs(tp - prev) / prev >= (double)a.mod_thresh) rep = 1;
    }
    if (a.tpwr_out) *a.tpwr_out = tp;
    if (a.status) a.status[0] = rep;
  }
}

// flag (:459-474) then make_ts (:414-453), and for the beam's last CTA
// simple_tsflag (:612-653) and flagts (:479-494).  Grid (row chunks of
// kApplyRows, beams).  The flagged channels' 16-byte chunks are listed once
// per CTA (ballot scan, channel order); L lanes share a row, L the power of
// two covering the listed chunks (at most 32), so a few flagged channels
// cost a few sectors per row and a fully flagged row is read once,
// coalesced.  Each listed chunk is read, its flagged channels set to the
// level MN * bpwr (clean mode) and written back, and
//   ts = (row sum from the statistics pass + sum over flagged channels of
//         (level - x)) / nchan,
// which for uint8 is a sum of exact integers, so it equals the reference's
// float tree sum / NCHAN_P bit for bit.  Each CTA then counts itself in; the
// beam's last one takes the median and MAD (lower medians, by radix select)
// of the first ts_base samples, flags rows with ts - med > TsThr * MAD
// (one-sided) and, in clean mode, sets channels [guard, nchan - guard) of
// the flagged rows to the level.  A block the modulation check replaced
// gets the noise block in every beam (clean mode, :1323-1324) and zero
// masks; its ts keeps the raw row sums.
template <typename E>
__global__ void __launch_bounds__(flag::kApplyThreads) flag_apply_kernel(FlagArgs a) {
  constexpr int ES = (int)sizeof(E), EPC = 16 / ES;   // elements per 16-byte chunk
  const int b = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int C = a.nchan, G = a.guard, T = a.ntime, NCH = C / EPC;
  const int t_begin = blockIdx.x * flag::kApplyRows;
  const int t_end = min(T, t_begin + flag::kApplyRows);
  constexpr int nw = flag::kApplyThreads / 32;
  extern __shared__ __align__(16) uint32_t ash[];
  uint32_t *chk = ash;                                            // [NCH]
  float *tsb = reinterpret_cast<float *>(ash + NCH);              // [ts_base]
  float *tmp = tsb + a.ts_base;                                   // [ts_base]
  __shared__ uint32_t hist[256], sel[2];
  __shared__ int nact_sh, last_sh;
  __shared__ float lev_sh, lvl_sh;
  E *xw = a.clean ? elem_out<E>(a) : nullptr;
  uint8_t *mb = a.tsmask + (int64_t)b * T;
  if (a.status && a.status[0]) {   // replaced by noise
    const E *nz = static_cast<const E *>(a.noise);
    if (xw && nz) {
      const uint4 *src = reinterpret_cast<const uint4 *>(nz + (int64_t)t_begin * C);
      uint4 *dst = reinterpret_cast<uint4 *>(xw + ((int64_t)b * T + t_begin) * C);
      const int64_t nv = (int64_t)(t_end - t_begin) * C / EPC;
      for (int64_t i = tid; i < nv; i += flag::kApplyThreads) dst[i] = src[i];
    }
    for (int t = t_begin + tid; t < t_end; t += flag::kApplyThreads) mb[t] = 0;
    if (blockIdx.x == 0)
      for (int c = tid; c < C; c += flag::kApplyThreads) a.chanmask[b * C + c] = 0;
    if (blockIdx.x == 0 && b == 0 && tid == 0 && a.counts) {
      a.counts[0] = 0;
      a.counts[1] = 0;
    }
    return;
  }
  if (tid == 0) {   // calc_bpwr (:759-769): float sum over every channel, in order
    float lvl = a.bpwr ? a.bpwr[b] : 1.0f;
    if (a.pwr && a.bpwr) {
      float acc = 0.0f;
      for (int c = 0; c < C; ++c) acc += a.spec[b * C + c];
      lvl = (float)(((double)acc / (double)(C - 2 * G)) / (double)a.mn);
    }
    lvl_sh = lvl;
    lev_sh = a.mn * lvl;
  }
  if (warp == 0) {   // the chunks holding flagged channels: index | element mask << 16
    int base = 0;
    for (int k0 = 0; k0 < NCH; k0 += 32) {
      const int k = k0 + lane;
      uint32_t m = 0u;
      if (k < NCH)
        for (int e = 0; e < EPC; ++e) m |= (uint32_t)a.chanmask[b * C + k * EPC + e] << e;
      const uint32_t bal = __ballot_sync(0xffffffffu, m != 0u);
      if (m) chk[base + __popc(bal & ((1u << lane) - 1u))] = (uint32_t)k | (m << 16);
      base += __popc(bal);
    }
    if (lane == 0) nact_sh = base;
  }
  __syncthreads();
  __shared__ double corr_sh[flag::kApplyRows];   // per row: sum over flagged channels of (level - x)
  const int nact = nact_sh;
  const E re = repl_elem<E>(lev_sh);
  const float rf = (float)re;
  int L = 1;
  while (L < nact && L < 32) L <<= 1;
  const int rpw = 32 / L, sub = lane & (L - 1);
  const E *xin = (a.spec0 && elem_out<E>(a)) ? elem_out<E>(a) : elem_in<E>(a);
  for (int i = tid; i < flag::kApplyRows; i += flag::kApplyThreads) corr_sh[i] = 0.0;
  __syncthreads();
  // a lane keeps one chunk (and its element masks) while its warp goes down
  // the rows, kApplyUnroll row groups of loads in flight
  const int64_t rowlen = C / EPC;              // 16-byte words
  const uint4 *xrow = reinterpret_cast<const uint4 *>(xin + (int64_t)b * T * C);
  uint4 *wrow = xw ? reinterpret_cast<uint4 *>(xw + (int64_t)b * T * C) : nullptr;
  for (int i0 = 0; i0 < nact; i0 += L) {
    const bool have = i0 + sub < nact;
    const uint32_t ce = have ? chk[i0 + sub] : 0u;
    const int k = (int)(ce & 0xFFFFu);
    const uint32_t m = ce >> 16;
    uint32_t mk[4];                            // bit masks of the flagged elements, per word
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      if constexpr (ES == 4) {
        mk[w] = (m >> w) & 1u ? 0xFFFFFFFFu : 0u;
      } else {
        const uint32_t n4 = (m >> (4 * w)) & 15u;
        mk[w] = (((n4 & 1u) | ((n4 & 2u) << 7) | ((n4 & 4u) << 14) | ((n4 & 8u) << 21)) * 255u);
      }
    }
    uint32_t rw;                               // the level in every element of a word
    if constexpr (ES == 4) rw = __float_as_uint(re); else rw = (uint32_t)re * 0x01010101u;
    for (int r0 = t_begin + warp * rpw; r0 < t_end; r0 += flag::kApplyUnroll * nw * rpw) {   // uniform
      uint4 v[flag::kApplyUnroll];
#pragma unroll
      for (int u = 0; u < flag::kApplyUnroll; ++u) {
        const int t = r0 + u * nw * rpw + lane / L;
        if (have && t < t_end) v[u] = xrow[(int64_t)t * rowlen + k];
      }
#pragma unroll
      for (int u = 0; u < flag::kApplyUnroll; ++u) {
        const int t = r0 + u * nw * rpw + lane / L;
        const bool on = have && t < t_end;
        uint32_t x[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
        double corr = 0.0;
        if (on) {
          if constexpr (ES == 4) {
#pragma unroll
            for (int w = 0; w < 4; ++w)
              if (mk[w]) corr += (double)(rf - __uint_as_float(x[w]));
          } else {
            uint32_t old = 0u;
#pragma unroll
            for (int w = 0; w < 4; ++w) old = __dp4a(x[w] & mk[w], 0x01010101u, old);
            corr = (double)((int)re * __popc(m) - (int)old);
          }
          if (wrow)
            wrow[(int64_t)t * rowlen + k] =
                make_uint4((x[0] & ~mk[0]) | (rw & mk[0]), (x[1] & ~mk[1]) | (rw & mk[1]),
                           (x[2] & ~mk[2]) | (rw & mk[2]), (x[3] & ~mk[3]) | (rw & mk[3]));
        }
        if constexpr (ES == 4) {
          for (int o = L >> 1; o > 0; o >>= 1) corr += __shfl_xor_sync(0xffffffffu, corr, o);
        } else {                               // whole numbers: 32-bit sums
          int ci = (int)corr;
          for (int o = L >> 1; o > 0; o >>= 1) ci += __shfl_xor_sync(0xffffffffu, ci, o);
          corr = (double)ci;
        }
        if (sub == 0 && t < t_end) corr_sh[t - t_begin] += corr;
      }
    }
  }
  __syncthreads();
  // the channel-mean series of the chunk's rows
  for (int t = t_begin + tid; t < t_end; t += flag::kApplyThreads) {
    double rsum;
    if (a.nslab == 1) {
      rsum = a.ts[(int64_t)b * T + t];
    } else {
      rsum = 0.0;
#pragma unroll 8
      for (int s = 0; s < a.nslab; ++s) rsum += a.rowsum[((int64_t)b * a.nslab + s) * T + t];
    }
    a.ts[(int64_t)b * T + t] = (float)((rsum + corr_sh[t - t_begin]) / C);
  }
  // the beam's last CTA makes the time-series decisions
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    last_sh = atomicAdd(a.ctr + a.nbeam + b, 1) == (int)gridDim.x - 1;
    if (blockIdx.x == 0 && a.pwr && a.bpwr) a.bpwr[b] = lvl_sh;
  }
  __syncthreads();
  if (!last_sh) return;
  __threadfence();
  if (!a.tsflag) {
    for (int t = tid; t < T; t += flag::kApplyThreads) mb[t] = 0;
    return;
  }
  const float *tb = a.ts + (int64_t)b * T;
  for (int i = tid; i < a.ts_base; i += flag::kApplyThreads) tsb[i] = tb[i];
  __syncthreads();
  const int kmed = (a.ts_base + 1) / 2 - 1;   // lower median
  const float med =
      grp_radix_select(tsb, a.ts_base, kmed, hist, sel, tid, flag::kApplyThreads, 1);
  for (int i = tid; i < a.ts_base; i += flag::kApplyThreads) tmp[i] = fabsf(tsb[i] - med);
  __syncthreads();
  const float mad =
      grp_radix_select(tmp, a.ts_base, kmed, hist, sel, tid, flag::kApplyThreads, 1);
  const float lim = a.ts_thresh * mad;
  int nts = 0;
  // 32 rows per warp and step, eight steps of loads in flight; a warp sets its
  // own flagged rows from its lanes' votes (read back from memory row by row
  // they took most of this kernel: 500 of 700 us for 16,384 rows)
  for (int t0 = 32 * warp; t0 < T; t0 += 8 * 32 * nw) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int t = t0 + u * 32 * nw + lane;
      v[u] = t < T ? __ldcg(tb + t) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int t = t0 + u * 32 * nw + lane;
      const bool f = t < T && (v[u] - med) > lim;
      if (t < T) mb[t] = f ? 1 : 0;
      uint32_t votes = __ballot_sync(0xffffffffu, f);
      if (lane == 0) nts += __popc(votes);
      if (!xw) continue;
      while (votes) {
        const int i = __ffs(votes) - 1;
        votes &= votes - 1u;
        E *row = xw + ((int64_t)b * T + (t - lane + i)) * C;
        for (int c = G + lane; c < C - G; c += 32) row[c] = re;
      }
    }
  }
  if (nts && a.counts) atomicAdd(a.counts + 1, nts);
}

// fix_zspec (:114-170) over naver blocks of history: per (beam, channel),
// the value whose count of other values <= it equals naver / 2 (ties
// resolve to one value); if no value has that count the first block's is
// kept, as the kernel leaves s0[block_id] unwritten then.
__global__ void flag_zspec_kernel(const float *hs, const float *hv, int naver, int bc, float *s0,
                                  float *v0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= bc) return;
  const int place = naver / 2;
  for (int which = 0; which < 2; ++which) {
    const float *h = which ? hv : hs;
    float out = h[i];
    for (int k = 0; k < naver; ++k) {
      const float x = h[(int64_t)k * bc + i];
      int ct = 0;
      for (int j = 0; j < naver; ++j)
        if (j != k && h[(int64_t)j * bc + i] <= x) ++ct;
      if (ct == place) out = x;
    }
    (which ? v0 : s0)[i] = out;
  }
}

// median_calc (:771-798): per channel the lower median over beams
// (sorted[(nbeam + 1) / 2 - 1]; beam 31 of 64 in the reference), then
// broadcast to every beam.  One thread per channel.
__global__ void flag_medcalc_kernel(float *arr0, float *arr1, int nbeam, int nchan) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nchan) return;
  const int k = (nbeam + 1) / 2 - 1;
  for (int which = 0; which < 2; ++which) {
    float *arr = which ? arr1 : arr0;
    float med = arr[c];
    for (int i = 0; i < nbeam; ++i) {
      const float x = arr[(int64_t)i * nchan + c];
      int r = 0;
      for (int j = 0; j < nbeam; ++j) {
        const float y = arr[(int64_t)j * nchan + c];
        r += (y < x) || (y == x && j < i);
      }
      if (r == k) med = x;
    }
    for (int i = 0; i < nbeam; ++i) arr[(int64_t)i * nchan + c] = med;
  }
}

// ---------------------------------------------------------------- launchers
bool flag_shape_ok(const FlagArgs &a) {
  const bool u8 = a.xu8 != nullptr;
  const int es = u8 ? 1 : 4;
  const void *x = u8 ? (const void *)a.xu8 : (const void *)a.x;
  if (!x || a.nchan < 4 || a.nchan > flag::kMaxChan || a.tbin < 1 || a.ntime < 1) return false;
  if ((a.nchan * es) % 16 || (reinterpret_cast<uintptr_t>(x) & 15u)) return false;
  // (pixel rows of at most 256 samples and 24 KB)
  if (a.pix_sum && (u8 || a.nchan > kFlagSlab || a.tds < 1 || a.tbin % a.tds ||
                    a.ntime % a.tbin || a.tds > 256 || (size_t)a.tds * a.nchan * 4 > 24576))
    return false;
  // uint8 sums are 32-bit within a range of rows (a bin, where there are at
  // least eight of them or they are short; else a warp's eighth of a bin or of
  // the tail).  A slab of g groups takes 32,768 * (256 / g) rows, an eighth of
  // them in passes of 32 / g rows: at most 49,152 rows per lane (20 groups)
  // where 2^32 / 255^2 is 66,051.
  const int cs = a.nchan < kFlagSlab ? a.nchan : kFlagSlab;
  const int P = flag::kStatThreads / (cs / 4);
  if (u8 && (a.ntime + P - 1) / P > 32768) return false;
  return true;
}

// The largest layout over the launch's slabs: the full slab width and, when
// nchan is not a multiple of it, the narrower last slab.
static size_t stats_smem(const FlagArgs &a, int es) {
  const int batch = es == 1 ? flag::batch<uint8_t>() : flag::batch<float>();
  const int bx = a.nchan < kFlagSlab ? a.nchan : kFlagSlab;
  const int rpw = 32 / (bx / 4);
  const size_t stage = ((size_t)batch * rpw * bx * es + 127) & ~(size_t)127;
  auto layout = [&](int cs) {
    const size_t acc = es == 1 ? 4 : 8;
    return flag::kWarps * (a.ring * stage + flag_rowbuf(cs, batch, rpw, (int)acc)) +
           acc * 2 * flag::kWarps * cs + sizeof(double) * cs + sizeof(float) * 2 * cs +
           (es == 1 && a.spec0 ? (size_t)256 * cs : 0);
  };
  size_t n = layout(bx);
  if (a.nchan > kFlagSlab && a.nchan % kFlagSlab) {
    const size_t l = layout(a.nchan % kFlagSlab);
    if (l > n) n = l;
  }
  // the channel decisions reuse the buffer: 12 nchan floats + nchan bytes
  const size_t dec = a.decide ? sizeof(float) * 12 * (size_t)a.nchan + a.nchan : 0;
  return n > dec ? n : dec;
}

// Time chunks per (slab, beam): enough CTAs to fill the GPU where there are
// few beams, none where a chunk would have fewer than eight bins (a warp then
// has part of a bin), or 1,024 rows of scaled uint8 (its table is 3 us of
// work).
int flag_chunks(int nbeam, int ntime, int nchan, int tbin, bool table) {
  const int64_t ctas = (int64_t)nbeam * ((nchan + kFlagSlab - 1) / kFlagSlab);
  const int nbins = ntime / tbin;
  int64_t n = flag::kTargetCtas / ctas;   // (one wave of CTAs)
  if (n > nbins / 8) n = nbins / 8;
  if (table && n > ntime / 1024) n = ntime / 1024;
  if (n > kFlagMaxChunks) n = kFlagMaxChunks;
  return n < 1 ? 1 : (int)n;
}

size_t flag_part_bytes(int nbeam, int ntime, int nchan, int tbin, bool table) {
  const int n = flag_chunks(nbeam, ntime, nchan, tbin, table);
  return n > 1 ? sizeof(double) * (size_t)nbeam * ((nchan + kFlagSlab - 1) / kFlagSlab) * n *
                     flag::kPartFields * kFlagSlab
               : 0;
}

// The error word of flagger launches made without a context
// (dsax_flag_noalloc, which has none to report to), one per device.
static __device__ int g_flag_err;
static int *flag_err_word() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  static std::atomic<int *> addr[64] = {};
  int *p = addr[dev].load(std::memory_order_acquire);
  if (!p) {
    void *q = nullptr;
    if (cudaGetSymbolAddress(&q, g_flag_err) != cudaSuccess) return nullptr;
    p = static_cast<int *>(q);
    addr[dev].store(p, std::memory_order_release);
  }
  return p;
}

// The filterbank as a 2-D tensor [nbeam * ntime rows][nchan] of its element
// type, boxes [brows rows][min(nchan, 128) channels], zero fill past nchan.
static int encode_filterbank_map(CUtensorMap *map, const FlagArgs &a, int brows) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return -1;
  const bool u8 = a.xu8 != nullptr;
  const int es = u8 ? 1 : 4;
  const int bx = a.nchan < kFlagSlab ? a.nchan : kFlagSlab;
  const cuuint64_t dims[2] = {(cuuint64_t)a.nchan, (cuuint64_t)a.nbeam * (cuuint64_t)a.ntime};
  const cuuint64_t strides[1] = {(cuuint64_t)a.nchan * es};
  const cuuint32_t box[2] = {(cuuint32_t)bx, (cuuint32_t)brows};
  const cuuint32_t estr[2] = {1u, 1u};
  void *base = u8 ? (void *)a.xu8 : (void *)a.x;
  const CUresult r = fn(map, u8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                        base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -1;
}

int launch_flag_stats(FlagArgs a, cudaStream_t st) {
  if (!flag_shape_ok(a)) return -1;
  const bool u8 = a.xu8 != nullptr;
  const int es = u8 ? 1 : 4;
  a.nslab = (a.nchan + kFlagSlab - 1) / kFlagSlab;
  if (a.nslab > 1 && !a.rowsum) return -1;
  a.nchunk = a.part && a.ctr ? flag_chunks(a.nbeam, a.ntime, a.nchan, a.tbin, u8 && a.spec0) : 1;
  if (a.nchunk > 1 && !a.decide &&
      cudaMemsetAsync(a.ctr, 0, sizeof(int) * flag_ctr_ints(a.nbeam, a.nchan), st) != cudaSuccess)
    return -2;
  if (!a.err) a.err = flag_err_word();
  if (!a.err) return -2;
  if (!a.wait_limit_ns) a.wait_limit_ns = 1000000000ull;
  const int bx = a.nchan < kFlagSlab ? a.nchan : kFlagSlab;
  const int brows = (u8 ? flag::batch<uint8_t>() : flag::batch<float>()) * (32 / (bx / 4));
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  if (encode_filterbank_map(&map, a, brows) != 0) return -2;
  // as deep a ring as lets two CTAs share an SM (20 channels, 256 beams x 512
  // samples: 47.7 us with one CTA per SM and three boxes, 34.3 with two CTAs)
  size_t sh = 0;
  for (a.ring = flag::kMaxRing; a.ring >= 2; --a.ring)
    if ((sh = stats_smem(a, es)) <= flag::kStatSmem || a.ring == 2) break;
  const dim3 grid(a.nslab * a.nchunk, a.nbeam);
  // full slabs, or the one slab of a 48-channel subband, have their own forms
  const int kind = a.nchan == 48 ? 1 : a.nchan % kFlagSlab == 0 && !a.pix_sum ? 2 : 0;
  void (*const kernels[3][3])(const CUtensorMap, FlagArgs) = {
      {flag_stats_kernel<uint8_t, false, 0>, flag_stats_kernel<uint8_t, false, 12>,
       flag_stats_kernel<uint8_t, false, 32>},
      {flag_stats_kernel<float, true, 0>, flag_stats_kernel<float, true, 12>, nullptr},
      {flag_stats_kernel<float, false, 0>, flag_stats_kernel<float, false, 12>,
       flag_stats_kernel<float, false, 32>}};
  const int row = u8 ? 0 : a.pix_sum ? 1 : 2;
  auto kernel = kernels[row][kind];
  static SmemAttrOnce attr[9];
  if (smem_attr_once(attr[3 * row + kind], kernel, 160 * 1024) != cudaSuccess) return -2;
  kernel<<<grid, flag::kStatThreads, sh, st>>>(map, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// The statistics pass (which ends with the channel decisions and the total
// power), then the row-chunked apply pass (whose last CTA per beam makes the
// time-series decisions): two launches on one stream.
int launch_flag(const FlagArgs &a0, cudaStream_t st) {
  FlagArgs a = a0;
  if (a.nchan > flag::kMaxChan || a.ts_base < 1 || a.ts_base > flag::kMaxTsBase ||
      a.ts_base > a.ntime)
    return -1;
  if (!a.ctr) return -1;
  a.ts_mean = 0;
  a.decide = 1;
  a.nslab = (a.nchan + kFlagSlab - 1) / kFlagSlab;
  if (cudaMemsetAsync(a.ctr, 0, sizeof(int) * (a.part ? flag_ctr_ints(a.nbeam, a.nchan)
                                                    : flag_ctr_chunk(a.nbeam)), st) != cudaSuccess)
    return -2;
  int rc = launch_flag_stats(a, st);
  if (rc != 0) return rc;
  const bool u8 = a.xu8 != nullptr;
  const int nch = a.nchan * (u8 ? 1 : 4) / 16;
  const size_t sh = sizeof(uint32_t) * nch + sizeof(float) * 2 * (size_t)a.ts_base;
  const dim3 grid((a.ntime + flag::kApplyRows - 1) / flag::kApplyRows, a.nbeam);
  if (u8)
    flag_apply_kernel<uint8_t><<<grid, flag::kApplyThreads, sh, st>>>(a);
  else
    flag_apply_kernel<float><<<grid, flag::kApplyThreads, sh, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int launch_flag_baseline(const float *hist_spec, const float *hist_var, int naver, int nbeam,
                         int nchan, float *spec0, float *var0, cudaStream_t st) {
  const int bc = nbeam * nchan;
  flag_zspec_kernel<<<(bc + 255) / 256, 256, 0, st>>>(hist_spec, hist_var, naver, bc, spec0, var0);
  flag_medcalc_kernel<<<(nchan + 127) / 128, 128, 0, st>>>(spec0, var0, nbeam, nchan);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace dsax

namespace dsax {
__device__ __forceinline__ float slogf(float v) { return copysignf(log1pf(fabsf(v)), v); }

// Learned-flagger input features of one beam (one CTA per beam) from the
// statistics pass: the plain flagger's four channel test statistics and its
// time-series statistic z, each scaled so that the plain rule fires at
// |z| = 1 (z > 1 for the one-sided pp and time-series rules), given as
// margins 10 (|z| - 1), plus the downsampled spectrogram.  F[b][h][c][8],
// log-compressed by slog(v) = sign(v) log(1 + |v|):
//   f0 (pixel mean - mu) / sigma * sqrt(tds)   f1 (pixel max - mu) / sigma
//   f2 10 (max over the pixel's samples of z_ts - 1)
//   f3 10 (|z_spec| - 1)   f4 10 (|z_var| - 1)   f5 10 (|z_max| - 1)
//   f6 10 (z_pp - 1)       f7 mean over the pixel's samples of z_ts
// mu, sigma: mean and standard deviation of the beam's samples (from the
// per-channel mean and variance).
__global__ void __launch_bounds__(2 * flag::kDecThreads) lf_stat_features_kernel(FlagArgs a, float *F,
                                                                            uint16_t *Fbf) {
  const int b = blockIdx.x;
  const int C = a.nchan, G = a.guard, T = a.ntime, n = C - 2 * G, tds = a.tds, H = T / tds;
  extern __shared__ float lsh[];
  float *dsh = lsh;                                    // [4 tests][3][C]: statistic, detrended, scratch
  float *z = dsh + 12 * C;                             // [4][C]
  float *tmp = z + 4 * C;                              // ts_base
  float *zt = tmp + a.ts_base;                         // T
  float *rmax = zt + T;                                // H
  float *rmean = rmax + H;                             // H
  __shared__ uint32_t hist[5][256], sel[5][2];
  __shared__ float mu_sd[2], ts_med_mad[2];
  const int tid = threadIdx.x, warp = tid >> 5;
  const float *tsb = a.ts + (int64_t)b * T;

  for (int i = tid; i < 4 * C; i += blockDim.x) {
    const int k = i / C, c = i - k * C;
    const float *src = k == 0 ? a.spec : k == 1 ? a.var : k == 2 ? a.maxs : a.pp;
    dsh[3 * C * k + c] = src[b * C + c];
    dsh[3 * C * k + C + c] = NAN;   // what a window without a median leaves
    z[i] = 0.0f;
  }
  for (int i = tid; i < a.ts_base; i += blockDim.x) zt[i] = tsb[i];
  __syncthreads();
  grp_detrend3(dsh, a, tid, blockDim.x);
  __syncthreads();
  // the four channel tests in four groups of 64 threads and the time series'
  // median and MAD in the other 256, all at once (one after the other by the
  // whole CTA, each with its barriers, they were half of this kernel)
  if (warp < 8) {
    const int k = warp >> 1, gtid = tid & 63, bid = 1 + k;
    float *sb = dsh + 3 * C * k, *corr = sb + C, *tm = corr + C;
    if (k < 3) {
      // channflag()'s test statistic: corr[j] / (thr * MAD), so the channel is
      // flagged exactly when |z| > 1 (z = +-1e6 when the MAD is 0 and corr is
      // not; 0 in the guard band)
      const float thr = k == 1 ? a.thresh + a.var_add : a.thresh;
      const float med = grp_select_call(corr, n, (n + 1) / 2 - 1, hist[k], sel[k], gtid, 64, bid);
      for (int i = gtid; i < n; i += 64) tm[i] = fabsf(corr[i] - med);
      named_bar(bid, 64);
      const float mad = grp_select_call(tm, n, (n + 1) / 2 - 1, hist[k], sel[k], gtid, 64, bid);
      for (int i = gtid; i < n; i += 64) {
        const float v = corr[i];
        z[k * C + G + i] = mad > 0.0f ? v / (thr * mad) : (v > 0.0f ? 1e6f : (v < 0.0f ? -1e6f : 0.0f));
      }
    } else {
      // simple_channflag(pp): one-sided, FBIN-channel mean against med + Thr/sqrt(FBIN) MAD
      const float med = grp_select_call(sb + G, n, (n + 1) / 2 - 1, hist[k], sel[k], gtid, 64, bid);
      for (int i = gtid; i < n; i += 64) tm[i] = fabsf(sb[G + i] - med);
      named_bar(bid, 64);
      const float mad = grp_select_call(tm, n, (n + 1) / 2 - 1, hist[k], sel[k], gtid, 64, bid);
      const float mythr = a.thresh / sqrtf((float)a.fbin);
      for (int j = G + gtid; j < C - G - a.fbin; j += 64) {
        float vv = 0.0f;
        for (int q = 0; q < a.fbin; ++q) vv += a.parity ? sb[j] : sb[j + q];
        vv = vv / (float)a.fbin - med;
        z[3 * C + j] = mad > 0.0f ? vv / (mythr * mad) : (vv > 0.0f ? 1e6f : (vv < 0.0f ? -1e6f : 0.0f));
      }
    }
  } else {   // simple_tsflag: median and MAD over the first ts_base samples
    const int gtid = tid - 256, gsize = (int)blockDim.x - 256, k = (a.ts_base + 1) / 2 - 1;
    const float med = grp_select_call(zt, a.ts_base, k, hist[4], sel[4], gtid, gsize, 5);
    for (int i = gtid; i < a.ts_base; i += gsize) tmp[i] = fabsf(zt[i] - med);
    named_bar(5, gsize);
    const float mad = grp_select_call(tmp, a.ts_base, k, hist[4], sel[4], gtid, gsize, 5);
    if (gtid == 0) {
      ts_med_mad[0] = med;
      ts_med_mad[1] = mad;
    }
  }
  __syncthreads();
  {
    const float med = ts_med_mad[0], mad = ts_med_mad[1];
    for (int t = tid; t < T; t += blockDim.x) {
      const float vv = tsb[t] - med;
      float zz = mad > 0.0f ? vv / (a.ts_thresh * mad) : (vv > 0.0f ? 1e6f : (vv < 0.0f ? -1e6f : 0.0f));
      zt[t] = a.tsflag ? zz : 0.0f;
    }
  }
  if (threadIdx.x < 32) {   // beam mean and variance over channels, one warp
    double s = 0.0, q = 0.0;
    for (int c = threadIdx.x; c < C; c += 32) {
      const double m = a.spec[b * C + c];
      s += m;
      q += (double)a.var[b * C + c] + m * m;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      q += __shfl_xor_sync(0xffffffffu, q, o);
    }
    if (threadIdx.x == 0) {
      const double mu = s / C;
      mu_sd[0] = (float)mu;
      mu_sd[1] = (float)sqrt(fmax(q / C - mu * mu, 1e-30));
    }
  }
  __syncthreads();
  for (int h = threadIdx.x; h < H; h += blockDim.x) {
    float mx = -INFINITY, sm = 0.0f;
    for (int r = 0; r < tds; ++r) {
      const float v = zt[h * tds + r];
      mx = fmaxf(mx, v);
      sm += v;
    }
    rmax[h] = mx;
    rmean[h] = sm / tds;
  }
  __syncthreads();
  const float mu = mu_sd[0], inv = 1.0f / mu_sd[1], kpix = sqrtf((float)tds);
  constexpr float kMargin = 10.0f;   // margins scaled so the rule's edge is steep
  // features that depend only on the channel (f3..f6) or only on the row
  // (f2, f7): once each, in place
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    z[c] = slogf(kMargin * (fabsf(z[c]) - 1.0f));
    z[C + c] = slogf(kMargin * (fabsf(z[C + c]) - 1.0f));
    z[2 * C + c] = slogf(kMargin * (fabsf(z[2 * C + c]) - 1.0f));
    z[3 * C + c] = slogf(kMargin * (z[3 * C + c] - 1.0f));
  }
  for (int h = threadIdx.x; h < H; h += blockDim.x) {
    rmax[h] = slogf(kMargin * (rmax[h] - 1.0f));
    rmean[h] = slogf(rmean[h]);
  }
  __syncthreads();
  float4 *Fb = F ? reinterpret_cast<float4 *>(F + (int64_t)b * H * C * 8) : nullptr;
  const float *ps = a.pix_sum + (int64_t)b * H * C;
  const float *pm = a.pix_max + (int64_t)b * H * C;
  const float invC = 1.0f / (float)C, invT = 1.0f / (float)tds;
  constexpr int kBatch = 4;   // pixel loads issued together
  for (int i0 = threadIdx.x; i0 < H * C; i0 += kBatch * blockDim.x) {
    float pv[kBatch], mv[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int i = i0 + k * blockDim.x;
      pv[k] = i < H * C ? ps[i] : 0.0f;
      mv[k] = i < H * C ? pm[i] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
    const int i = i0 + k * blockDim.x;
    if (i >= H * C) break;
    int h = __float2int_rz((float)i * invC);   // i / C, corrected (i < 2^24)
    h += (i - h * C >= C) - (i - h * C < 0);
    const int c = i - h * C;
    float4 f, g;
    f.x = slogf((pv[k] * invT - mu) * inv * kpix);
    f.y = slogf((mv[k] - mu) * inv);
    f.z = rmax[h];
    f.w = z[c];
    g.x = z[C + c];
    g.y = z[2 * C + c];
    g.z = z[3 * C + c];
    g.w = rmean[h];
    if (F) {
      Fb[2 * i] = f;
      Fb[2 * i + 1] = g;
    }
    if (Fbf) {
      uint4 o;
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o.x) : "f"(f.y), "f"(f.x));
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o.y) : "f"(f.w), "f"(f.z));
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o.z) : "f"(g.y), "f"(g.x));
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o.w) : "f"(g.w), "f"(g.z));
      // zero-bordered grid [B][H+2][C+2][8] read by the first conv layer
      reinterpret_cast<uint4 *>(Fbf)[((int64_t)b * (H + 2) + h + 1) * (C + 2) + c + 1] = o;
    }
    }
  }
}

int launch_lf_stat_features(const FlagArgs &a, float *F, uint16_t *Fbf, cudaStream_t st) {
  if (!a.pix_sum || a.tds < 1 || a.ntime % a.tds || a.nchan > flag::kLfMaxChan) return -1;
  const int H = a.ntime / a.tds;
  if (sizeof(float) * (6 * a.nchan + (a.ts_base > a.nchan ? a.ts_base : a.nchan) + a.ntime + 2 * H) >
      200 * 1024)
    return -1;
  const size_t sh = sizeof(float) * (16 * a.nchan + a.ts_base + a.ntime + 2 * H);
  static SmemAttrOnce attr;
  if (smem_attr_once(attr, lf_stat_features_kernel, 210 * 1024) != cudaSuccess) return -2;
  lf_stat_features_kernel<<<a.nbeam, 2 * flag::kDecThreads, sh, st>>>(a, F, Fbf);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace dsax

// ---------------------------------------------------------------------------
// Allocation-free variant of the plain flagger for callers that cannot call
// cudaMalloc (a process whose device memory is owned by another runtime or
// pool, a real-time thread that must not enter the allocator, or code that
// runs while a CUDA graph is being recorded by someone else).  The
// statistics live in this file-scope device array instead of a context
// buffer: every GPU that loads the library holds it until the process
// exits, every call shares it, and it keeps the last call's contents.
namespace dsax {

constexpr long long kNoAllocScratchFloats = 1572864;  // 6 MiB
static __device__ __align__(256) float g_flag_scratch[kNoAllocScratchFloats];

namespace {
constexpr int kMaxDevices = 64;
// device address of the array per device, looked up once; atomic because
// host threads may make their first call on a device concurrently (they
// store the same value)
std::atomic<float *> g_scratch_addr[kMaxDevices] = {};
}  // namespace

// Resolves the array's device address on the current device `dev` (once per
// device).  Returns nullptr on failure.
static float *noalloc_scratch(int dev) {
  if (dev < 0 || dev >= kMaxDevices) return nullptr;
  float *s = g_scratch_addr[dev].load(std::memory_order_acquire);
  if (!s) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_flag_scratch) != cudaSuccess) return nullptr;
    s = static_cast<float *>(p);
    g_scratch_addr[dev].store(s, std::memory_order_release);
  }
  return s;
}

}  // namespace dsax

extern "C" int dsax_flag_noalloc(const dsax_flag_params *p, const float *x, const float *oldspec,
                                 uint8_t *chanmask, uint8_t *tsmask, int *counts, void *stream) {
  using namespace dsax;
  if (!p || !x || !chanmask || !tsmask) return DSAX_ERR_ARG;
  const int B = p->nbeam, T = p->ntime, C = p->nchan;
  if (B < 1 || T < 1 || C < 1 || C > 128 || p->guard < 0 || C - 2 * p->guard < 1 ||
      p->filt < 1 || p->filt > C - 2 * p->guard || p->tbin < 1 || p->fbin < 1 ||
      p->ts_base < 1 || p->ts_base > T || p->ts_base > 4096 || p->nperm < 0 || p->nperm > 8)
    return DSAX_ERR_ARG;
  const long long nbc = (long long)B * C, nbt = (long long)B * T;
  // spec, var, max, pp, ts, the two flag counts, the launches' completion counters
  const long long need = 4 * nbc + nbt + 2 + 2 * (long long)B + 2;
  if (need > kNoAllocScratchFloats) return DSAX_ERR_ARG;   // beyond the fixed 6 MiB
  if (C % 4 || (reinterpret_cast<uintptr_t>(x) & 15u)) return DSAX_ERR_ARG;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return DSAX_ERR_CUDA;
  float *s = noalloc_scratch(dev);
  if (!s) return DSAX_ERR_CUDA;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  FlagArgs a{};
  a.x = x; a.oldspec = oldspec; a.chanmask = chanmask; a.tsmask = tsmask;
  a.nbeam = B; a.ntime = T; a.nchan = C;
  a.guard = p->guard; a.filt = p->filt; a.tbin = p->tbin; a.fbin = p->fbin;
  a.ts_base = p->ts_base; a.tsflag = p->tsflag; a.parity = p->parity;
  a.thresh = p->thresh; a.var_add = p->var_add; a.ts_thresh = p->ts_thresh;
  a.nperm = p->nperm;
  for (int i = 0; i < p->nperm; ++i) a.perm[i] = p->perm[i];
  a.spec = s; a.var = s + nbc; a.maxs = s + 2 * nbc; a.pp = s + 3 * nbc; a.ts = s + 4 * nbc;
  a.counts = reinterpret_cast<int *>(s + 4 * nbc + nbt);
  a.ctr = a.counts + 2;
  // time chunks where the array has room for their counters and partial results
  const long long nctr = (long long)flag_ctr_ints(B, C);
  const long long opart = (4 * nbc + nbt + 2 + nctr + 1) & ~1ll;
  const size_t npart = flag_part_bytes(B, T, C, p->tbin, false);
  if (npart && opart + (long long)(npart / 4) <= kNoAllocScratchFloats)
    a.part = reinterpret_cast<double *>(s + opart);
  // the counters accumulate with atomics: clear them (the array keeps the
  // previous call's values)
  if (cudaMemsetAsync(a.counts, 0, 2 * sizeof(int), st) != cudaSuccess) return DSAX_ERR_CUDA;
  if (launch_flag(a, st) != 0) return DSAX_ERR_CUDA;
  if (counts && cudaMemcpyAsync(counts, a.counts, 2 * sizeof(int), cudaMemcpyDeviceToDevice, st) !=
                    cudaSuccess)
    return DSAX_ERR_CUDA;
  return DSAX_OK;
}
