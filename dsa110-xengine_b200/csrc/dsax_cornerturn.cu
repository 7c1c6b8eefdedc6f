// dsax_cornerturn.cu -- the beam corner turn between the beamformer and the
// search-side flagger, as two device-side reorders around one all-to-all.
//
// The reference does it over sockets: every subband node (dsaX_dbnic)
// transposes its beamformer output [t][256 beams][48 ch] into one
// [64 beams][t][48 ch] message per search node (src/dsaX_dbnic.c:84-152),
// and every search node (dsaX_nicdb) places the 16 subbands' messages at
// channel CHOFF/8 + chgroup*48 of its [64 beams][16384 t][1024 ch]
// filterbank (src/dsaX_nicdb.c:180-196).  Here a GPU per subband packs its
// beams into one contiguous chunk per destination (dsax_ct_pack), an NCCL
// all-to-all over NVLink moves the chunks (the caller's collective:
// dsax.dist.beam_corner_turn), and the destination places them into its
// filterbank (dsax_ct_unpack), which dsax_flag_clean then reads as uint8.
// Both reorders are byte moves of whole channel rows: HBM-bound, 16-byte
// loads and stores when the row length allows.
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "../../include/dsax.h"
#include "dsax_ctx.h"
#include "dsax_internal.h"

namespace dsax {

// in [nt][nb][nc] -> out [ndest][nb/ndest][nt][nc]: one row of nc bytes per
// (t, beam); thread = one 16-byte (or 1-byte) piece.
template <int V>
__global__ void ct_pack_kernel(const uint8_t *__restrict__ in, uint8_t *__restrict__ out, int nt,
                               int nb, int nc, int ndest) {
  const int nbl = nb / ndest, pr = nc / V;
  const int64_t n = (int64_t)nt * nb * pr;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / pr;
    const int p = (int)(i - row * pr);
    const int t = (int)(row / nb), b = (int)(row - (int64_t)t * nb);
    const int d = b / nbl, j = b - d * nbl;
    const int64_t o = (((int64_t)d * nbl + j) * nt + t) * nc + (int64_t)p * V;
    if constexpr (V == 16)
      *reinterpret_cast<uint4 *>(out + o) = *reinterpret_cast<const uint4 *>(in + row * nc + p * V);
    else
      out[o] = in[row * nc + p];
  }
}

// recv [nsrc][nbl][nt][nc] -> fil[nbl][t0 + t][ch0 + s nc + k] of a
// filterbank with fil_nt samples and fil_nc channels per row.
//
// HBM-bound (every byte read and written once).  A CTA places some passes
// of rows of one beam; a thread owns one V-byte piece of the row (source s,
// piece p of its nc bytes) and a row phase, so its source and destination
// advance by constants and all divisions are done once per thread (one
// thread per piece of the whole array spent three 64-bit divisions on each 16
// bytes: 1,190 us for 16 x 64 x 16,384 x 48 bytes; this 271, a copy of as many
// bytes 245).  The stores are streaming ones (with default stores 597 us), the
// loads four in flight (eight 590).  Consecutive threads write
// consecutive pieces of a filterbank row; the pieces of a source's
// consecutive rows share lines, which the passes of one CTA find in L1.
// (Rows counted from the CTA's first one instead of absolutely: the same loop
// compiles to another order of the loads, 431 us.)
// A call of few CTAs gives each fewer passes: its time is the chain of one
// thread's rows (4 x 65,536 rows of 4 bytes: 16 passes 6.1 us, 4 passes 5.4).
constexpr int kCtThreads = 256, kCtUnroll = 4, kCtPasses = 16;
template <int V, int kPasses>
__global__ void __launch_bounds__(kCtThreads)
    ct_unpack_kernel(const uint8_t *__restrict__ recv, uint8_t *__restrict__ fil, int nsrc, int nbl,
                     int nt, int nc, int fil_nt, int fil_nc, int t0, int ch0, int pieces) {
  using W = typename std::conditional<
      V == 16, uint4,
      typename std::conditional<V == 8, uint2,
                                typename std::conditional<V == 4, uint32_t, uint8_t>::type>::type>::type;
  const int pr = nc / V;
  const int width = min(pieces, kCtThreads);          // pieces of a row per pass
  const int phases = kCtThreads / width;              // rows of a pass
  const int ph = (int)threadIdx.x / width, lane = (int)threadIdx.x - ph * width;
  if (ph >= phases) return;
  const uint32_t r0 = blockIdx.x * (uint32_t)(kPasses * phases) + (uint32_t)ph;
  const uint32_t r1 = min((uint32_t)nt, (blockIdx.x + 1u) * (uint32_t)(kPasses * phases));
  for (int q = lane; q < pieces; q += width) {
    const int s = q / pr, p = q - s * pr;
    for (int j = blockIdx.y; j < nbl; j += gridDim.y) {
      const uint8_t *src = recv + (((int64_t)s * nbl + j) * nt + r0) * nc + (int64_t)p * V;
      uint8_t *dst = fil + ((int64_t)j * fil_nt + t0 + r0) * fil_nc + ch0 + (int64_t)q * V;
      const int64_t sstep = (int64_t)phases * nc, dstep = (int64_t)phases * fil_nc;
#pragma unroll 1
      for (uint32_t r = r0; r < r1; r += kCtUnroll * phases) {
        W v[kCtUnroll];
#pragma unroll
        for (int k = 0; k < kCtUnroll; ++k)
          if (r + k * phases < r1) v[k] = __ldg(reinterpret_cast<const W *>(src + k * sstep));
#pragma unroll
        for (int k = 0; k < kCtUnroll; ++k)
          if (r + k * phases < r1) __stcs(reinterpret_cast<W *>(dst + k * dstep), v[k]);
        src += kCtUnroll * sstep;
        dst += kCtUnroll * dstep;
      }
    }
  }
}

}  // namespace dsax

using namespace dsax;

extern "C" int dsax_ct_pack(dsax_ctx *c, const uint8_t *beams, int nt, int nb, int nc, int ndest,
                            uint8_t *send) {
  if (!c || !beams || !send || nt < 1 || nb < 1 || nc < 1 || ndest < 1 || nb % ndest)
    return DSAX_ERR_ARG;
  DeviceGuard g(c->device);
  const bool v16 = nc % 16 == 0 && aligned16(beams) && aligned16(send);
  const int64_t n = (int64_t)nt * nb * (v16 ? nc / 16 : nc);
  const int grid = (int)((n + 255) / 256 < 8 * (int64_t)c->num_sms ? (n + 255) / 256
                                                                     : 8 * (int64_t)c->num_sms);
  if (v16)
    ct_pack_kernel<16><<<grid, 256, 0, c->stream>>>(beams, send, nt, nb, nc, ndest);
  else
    ct_pack_kernel<1><<<grid, 256, 0, c->stream>>>(beams, send, nt, nb, nc, ndest);
  return cuda_check(c, cudaGetLastError(), "corner-turn pack");
}

extern "C" int dsax_ct_unpack(dsax_ctx *c, const uint8_t *recv, int nsrc, int nbl, int nt, int nc,
                              uint8_t *fil, int fil_nt, int fil_nc, int t0, int ch0) {
  if (!c || !recv || !fil || nsrc < 1 || nbl < 1 || nt < 1 || nc < 1 || t0 < 0 || ch0 < 0 ||
      t0 + nt > fil_nt || ch0 + nsrc * nc > fil_nc)
    return DSAX_ERR_ARG;
  DeviceGuard g(c->device);
  // the widest piece that every row start and source step is a multiple of
  const uint64_t al = (uint64_t)nc | (uint64_t)fil_nc | (uint64_t)ch0 |
                      (uint64_t)reinterpret_cast<uintptr_t>(recv) |
                      (uint64_t)reinterpret_cast<uintptr_t>(fil);
  const int V = al % 16 == 0 ? 16 : al % 8 == 0 ? 8 : al % 4 == 0 ? 4 : 1;
  const int pieces = nsrc * (nc / V);
  const int width = pieces < kCtThreads ? pieces : kCtThreads;
  // (two CTAs per SM, or fewer passes)
  const int phases = kCtThreads / width;
  auto blocks = [&](int passes) { return (nt - 1) / (passes * phases) + 1; };
  const int passes = (int64_t)blocks(kCtPasses) * nbl < 2 * c->num_sms ? kCtUnroll : kCtPasses;
  const dim3 grid(blocks(passes), nbl < 65535 ? nbl : 65535);
  const bool few = passes != kCtPasses;
  auto kernel = V == 16  ? (few ? ct_unpack_kernel<16, kCtUnroll> : ct_unpack_kernel<16, kCtPasses>)
                : V == 8 ? (few ? ct_unpack_kernel<8, kCtUnroll> : ct_unpack_kernel<8, kCtPasses>)
                : V == 4 ? (few ? ct_unpack_kernel<4, kCtUnroll> : ct_unpack_kernel<4, kCtPasses>)
                         : (few ? ct_unpack_kernel<1, kCtUnroll> : ct_unpack_kernel<1, kCtPasses>);
  kernel<<<grid, kCtThreads, 0, c->stream>>>(recv, fil, nsrc, nbl, nt, nc, fil_nt, fil_nc, t0, ch0,
                                             pieces);
  return cuda_check(c, cudaGetLastError(), "corner-turn unpack");
}
