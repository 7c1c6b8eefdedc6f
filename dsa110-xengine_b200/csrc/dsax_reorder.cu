// dsax_reorder.cu -- the packet corner turn of src/dsaX_reorder_raw.c
// massage() (:153-169) on the GPU: captured [pkt][nant_in][nchan][2 t][2 pol]
// -> frequency rows of 128 bytes [64 ant][2 pol], one packed 4+4-bit byte per
// sample, padded antennas zero (the reference leaves them as the ring
// buffer's previous bytes), either in xGPU order [pkt][2 nchan] or as one
// stream per frequency [2 nchan][pkt]; and the channel-major order
// [nchan][pkt][64][2 t][2 pol].
#include <cstdint>
#include <cuda_runtime.h>

#include "dsax_internal.h"

namespace dsax {

namespace reorder {
constexpr int kPkt = 4;          // packets per CTA
constexpr int kChan = 32;        // channels per CTA (128 bytes of each antenna row)
constexpr int kThreads = 256;
constexpr int kUnits = kPkt * 32 * (kChan / 4) / kThreads;   // antenna pairs x 4 channels per thread
}  // namespace reorder

// HBM-bound: every byte is read and written once.  A thread loads the same
// four channels of two neighbouring antennas (two 16-byte loads, kUnits pairs
// in flight), and one prmt per word puts the two antennas' two pols of a time
// slot side by side, so a shared-memory row is already an output row; its
// 16-byte chunks are XORed with the channel quad, which keeps the 4-byte
// stores (8 quads x 4 pairs) and the 16-byte loads (a row of 8 chunks) free
// of bank conflicts.  A warp then writes four packets of one frequency (512
// contiguous bytes in a stream, four rows in xGPU order).  Output row (freq,
// pkt) at freq * fstride + pkt * pstride.
__global__ void __launch_bounds__(reorder::kThreads)
    reorder_kernel(const uint8_t *__restrict__ in, uint8_t *__restrict__ out, int npkt, int nant_in,
                   int nchan, int64_t pstride, int64_t fstride) {
  using namespace reorder;
  __shared__ __align__(16) uint32_t W[2 * kChan * kPkt * 32];   // [2 chan + t][pkt][128 B]
  const int c0 = blockIdx.x * kChan, p0 = blockIdx.y * kPkt;
  const int nc = min(kChan, nchan - c0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cq = lane & 7, ps = lane >> 3;          // channel quad, pair within the octet
  uint4 v[kUnits][2];
#pragma unroll
  for (int i = 0; i < kUnits; ++i) {
    const int r = warp + i * (kThreads / 32);       // (packet, octet)
    const int p = p0 + (r >> 3);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int ant = 8 * (r & 7) + 2 * ps + h;
      v[i][h] = make_uint4(0u, 0u, 0u, 0u);
      if (p < npkt && ant < nant_in && 4 * cq < nc) {
        const uint8_t *src = in + (((int64_t)p * nant_in + ant) * nchan + c0 + 4 * cq) * 4;
        if ((nchan & 3) == 0) {
          v[i][h] = __ldg(reinterpret_cast<const uint4 *>(src));
        } else {
          const uint32_t *s32 = reinterpret_cast<const uint32_t *>(src);
          v[i][h].x = s32[0];
          v[i][h].y = 4 * cq + 1 < nc ? s32[1] : 0u;
          v[i][h].z = 4 * cq + 2 < nc ? s32[2] : 0u;
          v[i][h].w = 4 * cq + 3 < nc ? s32[3] : 0u;
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kUnits; ++i) {
    const int r = warp + i * (kThreads / 32);
    const int pq = r >> 3;
    const uint32_t word = (uint32_t)(((((r & 7) ^ cq) & 7) << 2) + ps);
    const uint32_t *x = reinterpret_cast<const uint32_t *>(&v[i][0]);
    const uint32_t *y = reinterpret_cast<const uint32_t *>(&v[i][1]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {                   // channel 4 cq + k, words [t0p0, t0p1, t1p0, t1p1]
      uint32_t *w = W + ((2 * (4 * cq + k)) * kPkt + pq) * 32 + word;
      w[0] = __byte_perm(x[k], y[k], 0x5410u);
      w[kPkt * 32] = __byte_perm(x[k], y[k], 0x7632u);
    }
  }
  __syncthreads();
  const int o = lane & 7, pq = lane >> 3;
  if (p0 + pq >= npkt) return;
#pragma unroll
  for (int i = 0; i < 2 * kChan / (kThreads / 32); ++i) {
    const int fr = warp + i * (kThreads / 32);      // 2 chan + t within the CTA
    if (fr >= 2 * nc) break;
    const uint4 d = *reinterpret_cast<const uint4 *>(
        W + (fr * kPkt + pq) * 32 + (((o ^ (fr >> 3)) & 7) << 2));
    *reinterpret_cast<uint4 *>(out + (2 * c0 + fr) * fstride + (p0 + pq) * pstride + 16 * o) = d;
  }
}

static int launch_rows(const uint8_t *in, uint8_t *out, int npkt, int nant_in, int nchan,
                       int64_t pstride, int64_t fstride, cudaStream_t st) {
  using namespace reorder;
  if (npkt < 1 || nant_in < 1 || nant_in > 64 || nchan < 1) return -1;
  const dim3 grid((nchan + kChan - 1) / kChan, (npkt + kPkt - 1) / kPkt);
  if (grid.y > 65535) return -1;
  reorder_kernel<<<grid, kThreads, 0, st>>>(in, out, npkt, nant_in, nchan, pstride, fstride);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int launch_reorder(const uint8_t *in, uint8_t *out, int npkt, int nant_in, int nchan,
                   cudaStream_t st) {
  return launch_rows(in, out, npkt, nant_in, nchan, (int64_t)nchan * 256, 128, st);
}

int launch_reorder_freqmajor(const uint8_t *in, uint8_t *out, int npkt, int nant_in, int nchan,
                             cudaStream_t st) {
  return launch_rows(in, out, npkt, nant_in, nchan, 128, (int64_t)npkt * 128, st);
}

}  // namespace dsax

namespace dsax {

namespace reorder_cm {
constexpr int kPkt = 4;          // packets per CTA
constexpr int kChan = 32;        // channels per CTA
constexpr int kThreads = 256;
constexpr int kAStride = 65;     // words per channel row (64 antennas + 1 pad)
}  // namespace reorder_cm

// Captured [pkt][nant_in][nchan][4 B] -> channel-major [nchan][npkt][64][4 B]
// (padded antennas zero): each channel's samples become one contiguous
// stream, so the correlator can fetch a 64-packet stage with one bulk copy.
__global__ void __launch_bounds__(reorder_cm::kThreads) reorder_cm_kernel(
    const uint8_t *__restrict__ in, uint8_t *__restrict__ out, int npkt, int nant_in, int nchan) {
  using namespace reorder_cm;
  __shared__ uint32_t W[kPkt * kChan * kAStride];  // [pkt][chan][ant]
  const int c0 = blockIdx.x * kChan;
  const int p0 = blockIdx.y * kPkt;
  const int nc = min(kChan, nchan - c0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // load: lanes cover 8 x 16 B (32 channels) of 4 antenna rows; each warp
  // issues all of its rows' loads before the shared-memory stores, so eight
  // 16-byte loads per thread are in flight
  constexpr int kRows = kPkt * 16 / (kThreads / 32);   // rows per warp
  uint4 v[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int r = warp + i * (kThreads / 32);           // 4 pkts x 16 groups of 4 ants
    const int pq = r >> 4;
    const int a = 4 * (r & 15) + (lane >> 3);
    const int cq = lane & 7;
    const int p = p0 + pq;
    v[i] = make_uint4(0u, 0u, 0u, 0u);
    if (p < npkt && a < nant_in && 4 * cq < nc) {
      const uint8_t *src = in + (((int64_t)p * nant_in + a) * nchan + c0 + 4 * cq) * 4;
      if (4 * cq + 4 <= nc && ((nchan & 3) == 0)) {
        v[i] = __ldg(reinterpret_cast<const uint4 *>(src));
      } else {
        const uint32_t *s32 = reinterpret_cast<const uint32_t *>(src);
        v[i].x = s32[0];
        v[i].y = 4 * cq + 1 < nc ? s32[1] : 0u;
        v[i].z = 4 * cq + 2 < nc ? s32[2] : 0u;
        v[i].w = 4 * cq + 3 < nc ? s32[3] : 0u;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int r = warp + i * (kThreads / 32);
    const int pq = r >> 4;
    const int a = 4 * (r & 15) + (lane >> 3);
    const int cq = lane & 7;
    uint32_t *w = W + (pq * kChan + 4 * cq) * kAStride + a;
    w[0] = v[i].x;
    w[kAStride] = v[i].y;
    w[2 * kAStride] = v[i].z;
    w[3 * kAStride] = v[i].w;
  }
  __syncthreads();
  // store: per channel, kPkt x 256 B contiguous; a warp writes one channel
  for (int c = warp; c < nc; c += kThreads / 32) {
    uint8_t *dst = out + ((int64_t)(c0 + c) * npkt + p0) * 256;
#pragma unroll
    for (int k = lane; k < kPkt * 16; k += 32) {   // 16-byte chunks
      const int pq = k >> 4, a = 4 * (k & 15);
      if (p0 + pq >= npkt) continue;
      const uint32_t *w = W + (pq * kChan + c) * kAStride + a;
      *reinterpret_cast<uint4 *>(dst + 16 * k) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

int launch_reorder_chanmajor(const uint8_t *in, uint8_t *out, int npkt, int nant_in, int nchan,
                             cudaStream_t st) {
  using namespace reorder_cm;
  if (npkt < 1 || nant_in < 1 || nant_in > 64 || nchan < 1) return -1;
  dim3 grid((nchan + kChan - 1) / kChan, (npkt + kPkt - 1) / kPkt);
  if (grid.y > 65535) return -1;
  reorder_cm_kernel<<<grid, kThreads, 0, st>>>(in, out, npkt, nant_in, nchan);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace dsax
