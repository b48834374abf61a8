// TMA-staged block SpMV (1x1, 2x2 and 3x3 blocks): warp-specialised, persistent.
//
// The block rows are cut into tiles of consecutive rows (at most kBlocks
// off-diagonal blocks and kRows rows each; tile table built on the host from
// the pattern). A persistent grid (one CTA per SM) takes tiles round-robin. In
// each CTA one producer warp streams a tile's off-diagonal values, block
// columns, diagonal blocks and row offsets - four contiguous byte ranges,
// rounded out to 16 bytes - into a double-buffered shared-memory ring with
// cp.async.bulk, completing on a "full" mbarrier per stage; the consumer warps
// compute the tile's rows from shared memory (x gathered from global memory,
// read-only) and release the stage on an "empty" mbarrier. Every wait is
// bounded; on a timeout the kernel records DFM2G_ERR_WAIT_TIMEOUT and the
// producer still waits (bounded) for its copies in flight before exiting.
#pragma once

#include "rowkern.cuh"
#include "tma.cuh"

namespace dfm2g {

// Byte range [off, end) rounded out to 16 bytes: (aligned start, length).
__device__ __forceinline__ void round16(size_t off, size_t end, size_t &a, unsigned &len) {
  a = off & ~size_t(15);
  len = (unsigned)(((end + 15) & ~size_t(15)) - a);
}

// ---------------------------------------------------------------------------
// Component layout: lane B q + a of a consumer warp computes component a of
// row q of the warp's 32 / B rows, summing K_b[a][0..B-1] x_b over the row's
// blocks with no cross-lane reduction. A warp instruction then serves 10 rows of
// 3x3 blocks (16 of 2x2, 32 of 1x1), so the kernel issues a fraction of the
// instructions per row (and, in FP64, of the FP64 instructions) of a layout with
// a warp or eight lanes per row and a shuffle tree. Tiles hold 32 / B rows per
// consumer warp and are double-buffered; the tile's row offsets are staged
// with its values, block columns and diagonal blocks. FP32: 15 consumer warps
// (150-row tiles of 3x3 blocks), one CTA per SM. Tiles of 1x1 and 2x2 rows are
// sized for 16 blocks a row, which leaves the L1 cache room for x.
//
// FP64: a quarter of an SM issues one FP64 warp instruction per 64 cycles, so
// the product is bound by their number and by how evenly the warps cover the
// four quarters: eight consumer warps (80-row tiles), two per quarter, and three
// fused multiply-adds a block into six sums (component x block parity; two
// sums over whole blocks take a fourth instruction, the addition, per block).
// The rounding error is no larger: root mean square 0.299 against 0.305 units
// of 1e-16 |K||x| over 14-block rows that cancel, 0.180 against 0.212 on smooth
// vectors. 1x1 and 2x2 rows sum the same way in both types: over 14 terms 0.425
// units against eight lanes' sums and a tree's 0.418 (random ones), 0.256
// against 0.275 (smooth vectors), 0.503 against 0.551 (a dominant diagonal).
//
// One lane works through a row, so a long row is a long serial chain, of time
// and of roundings: patterns with a row of more than kLongest blocks take the
// kernels with a warp or eight lanes a row. 1x1 and 2x2: the two sums' error is
// 0.91 to 1.02 of the eight lanes' at 14 blocks, 0.91 to 1.16 at 24, up to 1.5 at
// 64 (four sums: 0.78 to 1.04 at 24, but 1.2 us more in 25 for the FP64 scalar
// product at 64^3); a 2,000-block row takes 106 us FP64 (52 ns a block) against
// 50. 3x3: a 1,400-block row takes 240 us FP64 against 35.
#ifndef DFM2G_SPMV_F32_CONSUMERS
#define DFM2G_SPMV_F32_CONSUMERS 15u  // FP32 tile: consumer warps (ten rows each)
#endif
#ifndef DFM2G_SPMV_F32_BLOCKS
#define DFM2G_SPMV_F32_BLOCKS 2304u  // FP32 tile: blocks at most
#endif
#ifndef DFM2G_SPMV_F32_STAGES
#define DFM2G_SPMV_F32_STAGES 2u  // FP32 ring stages
#endif
template <typename T, int B>
struct TileCfgC {
  static constexpr unsigned kConsumers = sizeof(T) == 8 ? 8u : DFM2G_SPMV_F32_CONSUMERS;
  static constexpr unsigned kThreads = 32u * (kConsumers + 1u);
  static constexpr unsigned kWarpRows = 32u / B;
  static constexpr unsigned kRows = kConsumers * kWarpRows;
  static constexpr unsigned kBlocks = B < 3 ? kRows * 16u : sizeof(T) == 8 ? 1424u : DFM2G_SPMV_F32_BLOCKS;
  static constexpr unsigned kLongest = B < 3 ? 16u : 1152u;
  static constexpr unsigned kStages = sizeof(T) == 8 ? 2u : DFM2G_SPMV_F32_STAGES;
  static constexpr unsigned kValBytes = kBlocks * B * B * sizeof(T) + 32;
  static constexpr unsigned kColBytes = kBlocks * 4 + 32;
  static constexpr unsigned kDiaBytes = (kRows * B * B * sizeof(T) + 32 + 15) / 16 * 16;
  static constexpr unsigned kRsBytes = ((kRows + 1) * 4 + 32 + 15) / 16 * 16;
  static constexpr unsigned kStageBytes = kValBytes + kColBytes + kDiaBytes + kRsBytes;
  static constexpr unsigned kBarBytes = 128;
  static constexpr size_t kSmem = kBarBytes + (size_t)kStages * kStageBytes;
  static_assert(kValBytes % 16 == 0 && kColBytes % 16 == 0 && kDiaBytes % 16 == 0 && kRsBytes % 16 == 0,
                "16-byte stage layout");
  static_assert(kSmem + 1024u <= 227u * 1024u, "fits one CTA's shared memory beside the reductions' words");
};

// Runs the pipeline over all tiles; epi(row, a, v) is called by the lane that
// computed component a of `row` (v = (K x)_{B row + a}). Must be called by all
// TileCfgC<T, B>::kThreads threads of the CTA; `smem` holds TileCfgC<T, B>::kSmem bytes.
template <typename T, int B, typename Epi>
__device__ __forceinline__ void spmv_tma_rows_c(const unsigned *__restrict__ tiles, unsigned ntiles,
                                                const unsigned *__restrict__ row_start,
                                                const unsigned *__restrict__ col, const T *__restrict__ vcrs,
                                                const T *__restrict__ vdia, const T *__restrict__ x, int *err,
                                                unsigned long long timeout_ns, unsigned char *smem, Epi &&epi) {
  using C = TileCfgC<T, B>;
  constexpr size_t BB = B * B, kBlk = BB * sizeof(T);  // values, bytes of one block
  uint64_t *full = reinterpret_cast<uint64_t *>(smem);
  uint64_t *empty = full + C::kStages;
  unsigned char *ring = smem + C::kBarBytes;
  const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  if (threadIdx.x == 0) {
    for (unsigned s = 0; s < C::kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], C::kConsumers);
    }
    mbar_fence_init();
  }
  __syncthreads();
  const unsigned G = gridDim.x;
  if (warp == C::kConsumers) {
    // producer: values, block columns, diagonal blocks and row offsets of a tile
    if (lane != 0) return;
    unsigned k = 0;
    for (unsigned t = blockIdx.x; t < ntiles; t += G, ++k) {
      const unsigned s = k % C::kStages;
      if (k >= C::kStages && !mbar_wait_bounded(&empty[s], ((k / C::kStages) - 1) & 1u, timeout_ns)) {
        atomicCAS(err, 0, DFM2G_ERR_WAIT_TIMEOUT);
        break;
      }
      const unsigned r0 = tiles[t], r1 = tiles[t + 1];
      const unsigned b0 = row_start[r0], b1 = row_start[r1];
      unsigned char *st = ring + (size_t)s * C::kStageBytes;
      size_t av, ac, ad, ar;
      unsigned lv, lc, ld, lr;
      round16((size_t)b0 * kBlk, (size_t)b1 * kBlk, av, lv);
      round16((size_t)b0 * 4, (size_t)b1 * 4, ac, lc);
      round16((size_t)r0 * kBlk, (size_t)r1 * kBlk, ad, ld);
      round16((size_t)r0 * 4, (size_t)(r1 + 1) * 4, ar, lr);
      mbar_arrive_expect_tx(&full[s], lv + lc + ld + lr);
      if (lv) tma_load_1d(st, reinterpret_cast<const unsigned char *>(vcrs) + av, lv, &full[s]);
      if (lc) tma_load_1d(st + C::kValBytes, reinterpret_cast<const unsigned char *>(col) + ac, lc, &full[s]);
      tma_load_1d(st + C::kValBytes + C::kColBytes, reinterpret_cast<const unsigned char *>(vdia) + ad, ld,
                  &full[s]);
      tma_load_1d(st + C::kValBytes + C::kColBytes + C::kDiaBytes,
                  reinterpret_cast<const unsigned char *>(row_start) + ar, lr, &full[s]);
    }
    const unsigned first = k > C::kStages ? k - C::kStages : 0u;
    for (unsigned j = first; j < k; ++j) mbar_wait_bounded(&full[j % C::kStages], (j / C::kStages) & 1u, timeout_ns);
    return;
  }
  const unsigned q = lane / B, a = lane - B * q;
  unsigned k = 0;
  for (unsigned t = blockIdx.x; t < ntiles; t += G, ++k) {
    const unsigned s = k % C::kStages;
    if (!mbar_wait_bounded(&full[s], (k / C::kStages) & 1u, timeout_ns)) {
      atomicCAS(err, 0, DFM2G_ERR_WAIT_TIMEOUT);
      break;
    }
    const unsigned r0 = tiles[t], r1 = tiles[t + 1];
    const unsigned char *st = ring + (size_t)s * C::kStageBytes;
    const unsigned *rsv = reinterpret_cast<const unsigned *>(st + C::kValBytes + C::kColBytes + C::kDiaBytes +
                                                             (((size_t)r0 * 4) & 15));
    const unsigned b0 = rsv[0];
    const T *vv = reinterpret_cast<const T *>(st + (((size_t)b0 * kBlk) & 15));
    const unsigned *cv = reinterpret_cast<const unsigned *>(st + C::kValBytes + (((size_t)b0 * 4) & 15));
    const T *dv = reinterpret_cast<const T *>(st + C::kValBytes + C::kColBytes + (((size_t)r0 * kBlk) & 15));
    const unsigned i = r0 + warp * C::kWarpRows + q;
    if (lane < C::kWarpRows * B && i < r1) {
      const unsigned s0 = rsv[i - r0] - b0, s1 = rsv[i - r0 + 1] - b0;
      const T *d = dv + (size_t)(i - r0) * BB + a * B, *xi = x + (size_t)i * B;
      unsigned u = s0;
      if constexpr (sizeof(T) == 8 || B < 3) {
        constexpr unsigned W = B == 3 ? 2 : 4;  // blocks per step
        T e[B] = {}, o[B] = {};                 // sums over the blocks of either parity
        // the next step's x gathered under this step's products, the first
        // step's under the row's remainder
        T g[W * B] = {};
        auto gather = [&](unsigned k) {
#pragma unroll
          for (unsigned w = 0; w < W; ++w)
#pragma unroll
            for (unsigned c = 0; c < B; ++c) g[w * B + c] = __ldg(x + (size_t)cv[k + w] * B + c);
        };
        const unsigned rem = (s1 - s0) % W;
        if (s0 + rem < s1) gather(s0 + rem);
#pragma unroll
        for (unsigned w = 0; w + 1 < W; ++w) {
          if (w < rem) {
            const T *v = vv + (size_t)u * BB + a * B, *y = x + (size_t)cv[u] * B;
#pragma unroll
            for (unsigned c = 0; c < B; ++c) (w & 1 ? o : e)[c] += v[c] * __ldg(y + c);
            ++u;
          }
        }
        while (u < s1) {
          const T *v = vv + (size_t)u * BB + a * B;
          T h[W * B];
#pragma unroll
          for (unsigned k = 0; k < W * B; ++k) h[k] = g[k];
          u += W;
          if (u < s1) gather(u);
#pragma unroll
          for (unsigned w = 0; w < W; ++w)
#pragma unroll
            for (unsigned c = 0; c < B; ++c) (w & 1 ? o : e)[c] += v[w * BB + c] * h[w * B + c];
        }
        // the diagonal block, the largest terms, summed apart and added late: few
        // sums are rounded at its size
        T t = d[0] * __ldg(xi);
#pragma unroll
        for (unsigned c = 1; c < B; ++c) t += d[c] * __ldg(xi + c);
        T se = e[0], so = o[0];
#pragma unroll
        for (unsigned c = 1; c < B; ++c) se += e[c], so += o[c];
        epi(i, a, se + (so + t));
      } else {
        T acc0 = T(0), acc1 = T(0);
        for (; u + 1 < s1; u += 2) {
          const unsigned j0 = cv[u], j1 = cv[u + 1];
          const T *v0 = vv + (size_t)u * 9 + a * 3, *v1 = v0 + 9;
          const T *x0 = x + (size_t)j0 * 3, *x1 = x + (size_t)j1 * 3;
          acc0 += v0[0] * __ldg(x0) + v0[1] * __ldg(x0 + 1) + v0[2] * __ldg(x0 + 2);
          acc1 += v1[0] * __ldg(x1) + v1[1] * __ldg(x1 + 1) + v1[2] * __ldg(x1 + 2);
        }
        if (u < s1) {
          const T *v0 = vv + (size_t)u * 9 + a * 3, *x0 = x + (size_t)cv[u] * 3;
          acc0 += v0[0] * __ldg(x0) + v0[1] * __ldg(x0 + 1) + v0[2] * __ldg(x0 + 2);
        }
        acc1 += d[0] * __ldg(xi) + d[1] * __ldg(xi + 1) + d[2] * __ldg(xi + 2);
        epi(i, a, acc0 + acc1);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
  }
}

}  // namespace dfm2g
