// dsax_corr_fm.cu -- the correlator over frequency rows: one CTA per SM takes
// one frequency (2 * channel + time slot) after another, with two TMEM
// accumulators so that a frequency's triangle is written while the next one
// is being multiplied.
//
// Input: [frequency][npkt][64 ant][2 pol] (the corner turn of a captured
// block, or the REORDER-key block [npkt][frequency][64][2]): a packet's 128
// samples of a frequency are 128 consecutive bytes in both, so one TMA box
// [128 packets][128 bytes] is a stage, whatever the two strides.
//
// Arithmetic: as in dsax_corr.cu.  Per 128-packet stage two MN-major
// SWIZZLE_128B int8 tiles of 128 packets (K) x 128 rows (2 ant + pol), R and
// I, each holding 16 times the nibbles; R [R; I]^T (N = 256) and I I^T
// (N = 128, added to the first 128 columns) give Re and E = R I^T, all times
// 256.
//
// Roles: unpack warps 0-3 in two groups of two that take alternate stages
// (a stage is a chain of waits, loads, stores, fence and arrival of about
// 1,000 cycles against 768 of its MMAs, so two are in flight); epilogue warps
// 4-11, two per TMEM lane quarter; warp 12 issues the MMAs; warp 13 the TMA
// boxes.
//
// What bounds it: no one unit.  For the full block the MMAs alone take 46 us, the
// boxes alone 41, everything but the MMAs 47; together 62-65, with the tensor
// pipe active 69 % of the busy SMs' cycles and shared memory at 66 % of the L1's
// peak.  (A stage of 768 MMA cycles counts 640 wavefronts of operand reads and
// 508 of the unpack and the epilogue; the two together are more than the
// stage's 1,109 cycles, so they do not share one port.)  What is left is how
// well the roles' waits overlap.  (One CTA per channel with the epilogue between channels:
// 76.)  Stages of 64 packets 77 us, of 256 73 (half the ring); loads straight
// into registers instead of boxes 66.  The loops that one thread runs per
// stage (boxes, MMAs) keep ring positions as counters: with a division by the
// number of stages and modulo indices they took 0.3 us per stage.  Short
// blocks are bound by the epilogue, a chain of loads, shuffles and stores:
// four warps 39.8 us for 128 packets x 384 channels with the corner turn,
// eight 28.8 (with eight unpack warps beside them registers spill: 30.9).
//
// Epilogue: the warps of quarter q hold rows j = 16q..16q+15 (x 2 pols) and
// write the outputs (i, j) for their columns i >= j as conjugates, so that the
// lanes of a store cover consecutive j: 512 contiguous bytes per store instead
// of 16 separate 32-byte pieces.  The block i >= 48, j < 16 goes to quarter 3
// in row order, which leaves no quarter more than three 16 x 16 blocks, split
// between its two warps.  Im needs E and its transpose: the 32 x 32 blocks of E
// that are read transposed go through shared memory, six and then four (24 KB).
// When accumulating, a block's old values are on their way while the one before
// it is written (loaded where they are added: 253 us against 137 for the full
// block with the corner turn).
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "dsax_internal.h"
#include "dsax_ptx.cuh"
#include "dsax_tmap.h"

namespace dsax {

namespace corrfm {
constexpr int kPkt = 128;                        // packets per stage
constexpr uint32_t kTile = kPkt * 128;           // one operand tile (R or I)
constexpr uint32_t kOpBytes = 2 * kTile;
constexpr uint32_t kRawBytes = kPkt * 128;
constexpr int kGroups = 2, kGroupWarps = 2;      // unpack warps: groups x warps of a group
constexpr int kOpStages = 4, kRawStages = 4;
// a ring slot is always the same group's: a group that skipped a phase of its
// barrier could not tell the next one from it
static_assert(kGroups <= kOpStages && kGroups <= kRawStages && kOpStages % kGroups == 0 && kRawStages % kGroups == 0, "ring slots of one group");
constexpr int kUnpackWarps = kGroups * kGroupWarps;
constexpr int kEpiWarps = 8;                     // two per TMEM lane quarter
constexpr int kUnits = kPkt * 8 / (32 * kGroupWarps);   // 16-byte chunks per thread and stage
constexpr uint32_t kScratch = 6 * 32 * 32 * 4;   // six 32 x 32 blocks of E
constexpr int kWarpMma = kUnpackWarps + kEpiWarps, kWarpTma = kWarpMma + 1;
constexpr int kThreads = 32 * (kWarpTma + 1);
constexpr int kSmem = 1024 + kOpStages * kOpBytes + kRawStages * kRawBytes + kScratch;
static_assert(kSmem <= 232448 - 1024, "shared memory of one CTA per SM");
constexpr uint32_t kIdescN128 = umma_idesc(/*S32*/ 2, /*s8*/ 1, /*s8*/ 1, 128, 128) | kIdescMnMajor;
constexpr uint32_t kIdescN256 = umma_idesc(/*S32*/ 2, /*s8*/ 1, /*s8*/ 1, 128, 256) | kIdescMnMajor;
}  // namespace corrfm

// Position in a ring of N stages and the parity of its current phase.
template <int N>
struct Ring {
  uint32_t i, ph = 0;
  __device__ explicit Ring(int start) : i((uint32_t)start) {}
  __device__ void step(int n) {
    i += (uint32_t)n;
    if (i >= (uint32_t)N) {
      i -= (uint32_t)N;
      ph ^= 1u;
    }
  }
};

__device__ __forceinline__ float4 add4(float4 x, float4 y) {
  return make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
}

// kAcc: adds to vis instead of overwriting it.
template <bool kAcc>
__global__ void __launch_bounds__(corrfm::kThreads, 1)
    corr_fm_kernel(const __grid_constant__ CUtensorMap tmap, CorrArgs a) {
  using namespace corrfm;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kOpStages], empty_bar[kOpStages];
  __shared__ __align__(8) uint64_t rfull_bar[kRawStages], rempty_bar[kRawStages];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
  __shared__ __align__(8) uint64_t final_bar;      // every MMA of the CTA complete
  __shared__ uint32_t tmem_base_sh;
  __shared__ volatile int abort_sh;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nfreq = 2 * a.nchan;
  const int nf = (nfreq - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int nks = (a.npkt + kPkt - 1) / kPkt;
  const int ntot = nf * nks;                       // stages of the CTA
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *const gbase = smem_raw + (sbase - smem_u32(smem_raw));
  const uint32_t raw_base = sbase + kOpStages * kOpBytes;

  if (tid == 0) {
    for (int s = 0; s < kOpStages; ++s) {
      mbar_init(&full_bar[s], kGroupWarps);
      mbar_init(&empty_bar[s], 1);
    }
    for (int r = 0; r < kRawStages; ++r) {
      mbar_init(&rfull_bar[r], 1);
      mbar_init(&rempty_bar[r], kGroupWarps);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kEpiWarps);
    }
    mbar_init(&final_bar, 1);
    abort_sh = 0;
    mbar_fence_init();
  }
  if (warp == kWarpMma) {
    tmem_alloc(&tmem_base_sh, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_sh;
  if ((tmem & 0xFFFFu) != 0u) {
    if (tid == 0) atomicOr(a.err, DEV_ERR_TMEM);
    abort_sh = 1;
  }

  if (warp < kUnpackWarps) {
    // ------------------------------------------------------------ unpack
    const uint32_t o = (uint32_t)lane & 7u;
    const uint32_t p_thr = (uint32_t)((kPkt / kGroupWarps) * (warp % kGroupWarps) + (lane >> 3));
    const uint4 *rw = reinterpret_cast<const uint4 *>(gbase + kOpStages * kOpBytes);
    Ring<kRawStages> r(warp / kGroupWarps);
    Ring<kOpStages> s(warp / kGroupWarps);
#pragma unroll 1
    for (int G = warp / kGroupWarps; G < ntot; G += kGroups, r.step(kGroups), s.step(kGroups)) {
      bool ok = mbar_wait_bounded(&rfull_bar[r.i], r.ph, &abort_sh, a.err, DEV_ERR_WAIT_FULL,
                                  a.wait_limit_ns);
      if (!__all_sync(0xffffffffu, ok)) break;
      uint4 w[kUnits];
#pragma unroll
      for (int u = 0; u < kUnits; ++u) w[u] = rw[r.i * (kRawBytes / 16) + (p_thr + 4 * u) * 8 + o];
      ok = mbar_wait_bounded(&empty_bar[s.i], s.ph ^ 1u, &abort_sh, a.err, DEV_ERR_WAIT_EMPTY,
                             a.wait_limit_ns);
      if (!__all_sync(0xffffffffu, ok)) break;
      const uint32_t stage = sbase + s.i * kOpBytes;
#pragma unroll
      for (int u = 0; u < kUnits; ++u) {
        const uint32_t P = p_thr + 4u * u;
        const uint32_t d = stage + P * 128u + ((o ^ (P & 7u)) << 4);
        st_shared_v4(d, x16_lo(w[u].x), x16_lo(w[u].y), x16_lo(w[u].z), x16_lo(w[u].w));
        st_shared_v4(d + kTile, x16_hi(w[u].x), x16_hi(w[u].y), x16_hi(w[u].z), x16_hi(w[u].w));
      }
      // one fence orders the stores before the MMAs' operand reads and the raw
      // stage's loads before the next box (async proxy) that overwrites it
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&full_bar[s.i]);
        mbar_arrive(&rempty_bar[r.i]);
      }
    }
  } else if (warp < kWarpMma) {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3, hh = (warp - kUnpackWarps) >> 2;   // TMEM lane quarter, share
    uint32_t *E = reinterpret_cast<uint32_t *>(gbase + kOpStages * kOpBytes + kRawStages * kRawBytes);
    const int j = 16 * q + (lane >> 1), pj = lane & 1;
#pragma unroll 1
    for (int fi = 0; fi < nf; ++fi) {
      const int b = fi & 1;
      const int64_t f = (int64_t)blockIdx.x + (int64_t)fi * gridDim.x;
      float4 *const out = reinterpret_cast<float4 *>(a.vis + f * (2080 * 8));   // 16-byte units
      // accumulating: the old values of the warp's share of block (I, q), each
      // set on its way while the one before is written (or waited for)
      using Old = float4[kAcc ? 8 : 1];
      Old oa, ob;
      auto load_old = [&](int I, Old &o) {
        if constexpr (kAcc) {
#pragma unroll
          for (int ii = 0; ii < 8; ++ii) {
            const int i = 16 * I + 8 * hh + ii;
            if (j <= i) o[ii] = out[i * (i + 1) + 2 * j + pj];
          }
        }
      };
      load_old(q, oa);
      bool ok = mbar_wait_bounded(&acc_full[b], (uint32_t)(fi >> 1) & 1u, &abort_sh, a.err,
                                  DEV_ERR_WAIT_ACCUM, a.wait_limit_ns);
      tc_fence_after();
      ok = __all_sync(0xffffffffu, ok && !abort_sh);
      const uint32_t trow = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)b * 256u;
      // block column J of this warp's rows of E -> scratch block k; the column
      // is XORed with the row, so that the row-wise stores and column-wise
      // loads are conflict-free
      auto save = [&](int J, int k) {
        uint32_t ev[32];
        tmem_ld32(trow + 128u + 32u * J, ev);
        tmem_wait_ld();
        uint32_t *blk = E + k * 1024 + lane * 32;
#pragma unroll
        for (int e = 0; e < 32; ++e) blk[e ^ lane] = ev[e];
      };
      // outputs (i, j): j the lanes' rows, i the warp's half (hh) of the 16
      // antennas of block row I, with E of block (I, q) in scratch block k
      auto conj_block = [&](int I, int k, const Old &old) {
        const uint32_t *blk = E + k * 1024;
        uint32_t re[16], er[16];
        tmem_ld16(trow + 32u * I + 16u * hh, re);
        tmem_ld16(trow + 128u + 32u * I + 16u * hh, er);
        tmem_wait_ld();
#pragma unroll
        for (int ii = 0; ii < 8; ++ii) {
          const int i = 16 * I + 8 * hh + ii;
          const int n0 = 16 * hh + 2 * ii, n1 = n0 + 1;
          const int32_t en0 = (int32_t)blk[n0 * 32 + (lane ^ n0)];
          const int32_t en1 = (int32_t)blk[n1 * 32 + (lane ^ n1)];
          const float x0 = vis_re(re[2 * ii]), y0 = vis_im((int32_t)er[2 * ii] - en0);
          const float x1 = vis_re(re[2 * ii + 1]), y1 = vis_im((int32_t)er[2 * ii + 1] - en1);
          // the two pols of j (lanes 2j, 2j + 1): pj = 0 keeps pi = 0 and
          // sends pi = 1, pj = 1 the reverse, so each writes 16 bytes
          const float sx = __shfl_xor_sync(0xffffffffu, pj ? x0 : x1, 1);
          const float sy = __shfl_xor_sync(0xffffffffu, pj ? y0 : y1, 1);
          float4 v = pj ? make_float4(sx, sy, x1, y1) : make_float4(x0, y0, sx, sy);
          if (j <= i) {
            if constexpr (kAcc) v = add4(v, old[ii]);
            out[i * (i + 1) + 2 * j + pj] = v;
          }
        }
      };
      // Two rounds, no quarter with more than two blocks and then one:
      //   (0,0) (1,0) | (1,1) (2,1) | (2,2) | (3,3), then
      //   (2,0)       | (3,1)       | (3,2) | (3,0) in row order.
      // Scratch blocks of the first: E (q,q) in q, (1,0) in 4, (2,1) in 5.
      if (ok) {
        if (hh == 0) save(q, q);
        else if (q == 1 || q == 2) save(q - 1, 3 + q);
      }
      named_bar(1, 32 * kEpiWarps);
      if (ok) {
        if (q < 2) load_old(q + 1, ob);
        conj_block(q, q, oa);
        if (q < 2) conj_block(q + 1, 4 + q, ob);
      }
      float4 *const row = out + j * (j + 1) + 16 * hh + pj;   // quarter 3: row antenna `j`, eight columns
      if constexpr (kAcc) {
        if (q < 3) {
          load_old(q == 0 ? 2 : 3, oa);
        } else {
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) oa[jj] = row[2 * jj];
        }
      }
      named_bar(1, 32 * kEpiWarps);
      // the second: (2,0) in 0, (3,1) in 1, (3,2) in 2, (0,3) in 3
      if (ok) {
        if (q == 0 && hh == 0) save(3, 3);
        if (q == 2 && hh == 0) save(0, 0);
        if (q == 3) save(1 + hh, 1 + hh);
      }
      named_bar(1, 32 * kEpiWarps);
      if (ok) {
        if (q < 3) {
          conj_block(q == 0 ? 2 : 3, q, oa);
        } else {   // i = 48..63 (this warp's rows; `j` is that antenna), eight j of 0..15
          const uint32_t *blk = E + 3 * 1024;
          uint32_t re[16], er[16];
          tmem_ld16(trow + 16u * hh, re);
          tmem_ld16(trow + 128u + 16u * hh, er);
          tmem_wait_ld();
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) {
            const int n0 = 16 * hh + 2 * jj, n1 = n0 + 1;
            const int32_t e0 = (int32_t)blk[n0 * 32 + (lane ^ n0)];
            const int32_t e1 = (int32_t)blk[n1 * 32 + (lane ^ n1)];
            float4 v = make_float4(vis_re(re[2 * jj]), vis_im(e0 - (int32_t)er[2 * jj]),
                                   vis_re(re[2 * jj + 1]), vis_im(e1 - (int32_t)er[2 * jj + 1]));
            if constexpr (kAcc) v = add4(v, oa[jj]);
            row[2 * jj] = v;
          }
        }
      }
      // the accumulator goes back to the MMA warp, and the scratch is free
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[b]);
      named_bar(1, 32 * kEpiWarps);
    }
  } else if (warp == kWarpMma) {
    // ------------------------------------------------------------ UMMA issuer
    if (lane == 0) {
      bool go = true;
      Ring<kOpStages> s(0);
      const uint64_t d0 = umma_desc_mn128(sbase, kTile, 1024u);   // (addresses in 16-byte units)
#pragma unroll 1
      for (int fi = 0; fi < nf && go; ++fi) {
        const int b = fi & 1;
        if (!mbar_wait_bounded(&acc_empty[b], ((uint32_t)(fi >> 1) & 1u) ^ 1u, &abort_sh, a.err,
                               DEV_ERR_WAIT_ACCUM, a.wait_limit_ns))
          break;
        const uint32_t dre = tmem + (uint32_t)b * 256u;
#pragma unroll 1
        for (int ks = 0; ks < nks; ++ks, s.step(1)) {
          if (!mbar_wait_bounded(&full_bar[s.i], s.ph, &abort_sh, a.err, DEV_ERR_WAIT_FULL,
                                 a.wait_limit_ns)) {
            go = false;
            break;
          }
          tc_fence_after();
          const uint64_t dr = d0 + s.i * (kOpBytes >> 4), di = dr + (kTile >> 4);
#pragma unroll
          for (int kk = 0; kk < kPkt / 32; ++kk)   // R [R; I]^T, 32 packets (4 KB) each
            umma_i8(dre, dr + 256u * kk, dr + 256u * kk, kIdescN256, (ks | kk) != 0);
#pragma unroll
          for (int kk = 0; kk < kPkt / 32; ++kk)   // += I I^T into the first 128 columns
            umma_i8(dre, di + 256u * kk, di + 256u * kk, kIdescN128, 1u);
          umma_commit(&empty_bar[s.i]);
        }
        if (go) umma_commit(&acc_full[b]);
      }
      umma_commit(&final_bar);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ TMA loader
    if (lane == 0) {
      Ring<kRawStages> r(0);
      int issued = 0;
      bool go = true;
#pragma unroll 1
      for (int fi = 0; fi < nf && go; ++fi)
#pragma unroll 1
        for (int ks = 0; ks < nks; ++ks, ++issued, r.step(1)) {
          if (!mbar_wait_bounded(&rempty_bar[r.i], r.ph ^ 1u, &abort_sh, a.err, DEV_ERR_WAIT_EMPTY,
                                 a.wait_limit_ns)) {
            go = false;
            break;
          }
          mbar_arrive_expect_tx(&rfull_bar[r.i], kRawBytes);
          tma_load_3d(raw_base + r.i * kRawBytes, &tmap, 0, ks * kPkt,
                      (int)blockIdx.x + fi * (int)gridDim.x, &rfull_bar[r.i]);
        }
      // boxes still landing after an abort: wait for the last one issued to
      // each raw stage before the CTA exits
      volatile int no_abort = 0;
      for (int k = issued - kRawStages; k < issued; ++k)
        if (k >= 0)
          mbar_wait_bounded(&rfull_bar[k % kRawStages], (uint32_t)(k / kRawStages) & 1u, &no_abort,
                            a.err, DEV_ERR_WAIT_FULL, drain_limit(a.wait_limit_ns));
    }
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kWarpMma) {
    if (lane == 0) {
      volatile int no_abort = 0;
      mbar_wait_bounded(&final_bar, 0u, &no_abort, a.err, DEV_ERR_WAIT_ACCUM,
                        drain_limit(a.wait_limit_ns));
    }
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// The block as a 3-D uint8 tensor [frequency][packet][128 bytes] with the
// given strides; boxes of 128 packets of one frequency, zero past npkt.
int launch_correlate_freq(const CorrArgs &a, size_t pkt_stride, size_t freq_stride, cudaStream_t st) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return -2;
  CUtensorMap tmap;
  const cuuint64_t dims[3] = {128, (cuuint64_t)a.npkt, 2 * (cuuint64_t)a.nchan};
  const cuuint64_t strides[2] = {(cuuint64_t)pkt_stride, (cuuint64_t)freq_stride};
  const cuuint32_t box[3] = {128u, (cuuint32_t)corrfm::kPkt, 1u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  if (fn(&tmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t *>(a.in), dims, strides, box,
         estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return -2;
  static SmemAttrOnce attr[2];
  auto kernel = a.accumulate ? corr_fm_kernel<true> : corr_fm_kernel<false>;
  if (smem_attr_once(attr[a.accumulate ? 1 : 0], kernel, corrfm::kSmem) != cudaSuccess) return -2;
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm < 1)
    return -2;
  // as few CTAs as give every CTA the largest share (768 frequencies: 128
  // CTAs of six)
  const int nfreq = 2 * a.nchan, per = (nfreq + nsm - 1) / nsm;
  const unsigned grid = (unsigned)((nfreq + per - 1) / per);
  kernel<<<grid, corrfm::kThreads, corrfm::kSmem, st>>>(tmap, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace dsax
