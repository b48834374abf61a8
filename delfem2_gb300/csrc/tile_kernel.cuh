// Kernel of the tile-scheduled triangular sweeps (tiles.cu), 1x1, 2x2 and 3x3
// blocks, FP32 and FP64, over the rows of the sweep's triangle:
//   backward           z_i = in_i - sum_j U'_ij z_j
//   forward, FP64      z_i = D_i^-1 in_i - sum_j (D_i^-1 L_ij) z_j
//   forward, FP32      z_i = D_i^-1 (in_i - sum_j L_ij z_j)
// In FP64 D^-1 is multiplied into the records when they are written (in FP64),
// which leaves three FP64 instructions out of a step's chain; the sweep's error
// is the unfolded one's (1.03e-16 against 1.04e-16 of quad precision at
// 40 x 37 x 43 voxels, within 1% either way for random 1x1 to 3x3 blocks). In
// FP32 the same would round D^-1 L and D^-1 apart and cost 16% in accuracy
// (9.5e-8 against 8.2e-8), so D^-1 is applied last there.
//
// One CTA sweeps one tile at a time, step by step (a step: the tile's rows of
// one local level). Its warps have three jobs:
//  - one producer warp streams each step's records and row list into a ring
//    of shared-memory slots (cp.async.bulk, one mbarrier per slot);
//  - HW fetch warps, each taking every HW-th step (the ring's length is a
//    multiple of HW, so that a slot is always the same warp's and it meets the
//    slot's phases in order), read the values the step needs from outside the tile (the right-hand side, and rows of other
//    tiles, polled in L2 until they are written) and store them in the slot;
//  - NW consumer warps compute. Every operand of theirs is then a row of
//    shared memory at a byte offset the record holds (the tile's own results, or
//    the slot's fetched rows), so their code is straight-line: no address,
//    no poll and no case distinction depends on where a row lives.
//
// Consumers: LPR = B S lanes work on a row; lane h B + a of the row sums
// component a over every S-th dependency, reading all B components of a
// dependency as one shared-memory vector, so no lane waits for another's
// products (S = 2: the two halves are added by one shuffle). G = 32 / LPR rows
// per warp and step. From barrier to barrier a step is: its operands, the
// products, the store; the next step's codes and values are read into
// registers meanwhile. One barrier per step: the consumers meet there with
// the fetch warps (bar.arrive), the next step's once its operands are in the
// slot, the one after's once its record has landed. Consumers never wait on
// an mbarrier themselves (a wait that succeeds at once costs about 100 cycles,
// the barrier 30).
//
// FP64 on GB300 issues one warp instruction per 64 cycles and SM quarter
// whatever the number of active lanes, so an FP64 step is split over four
// warps, one per quarter, six lanes a row: 13 FP64 instructions a step (14
// backward, which adds the right-hand side last).
#pragma once

#include "common.cuh"
#include "tma.cuh"

namespace dfm2g {

// Codes: the byte offset of an operand in shared memory (a row of the same
// tile), or kTiSlot + its offset in the slot's fetched rows.
constexpr unsigned kTiSlot = 0x80000000u;
constexpr unsigned kTiEnd = 0xFFFFFFFFu;
constexpr unsigned kTiMaxSlots = 12;
constexpr unsigned kTiGrabLead = 6;         // steps before a tile's end at which the next tile is taken
constexpr unsigned kTiAhead = 256u * 1024u; // bytes of records prefetched into L2 ahead of their copies
constexpr unsigned kTiDesc = 6;             // step descriptors the producer has in flight
constexpr unsigned kTiXsOff = 640;          // shared memory: barriers, slot descriptors and flags before it

// Lanes and rows of one consumer warp.
template <int B, int S>
struct TileLanes {
  static constexpr unsigned kLpr = B * S;          // lanes per row
  static constexpr unsigned kG = 32 / kLpr;        // rows per warp and step (a group)
  static constexpr unsigned kLanes = kG * kLpr;    // lanes in use
};

// Values per row in shared memory: FP32 3x3 rows are padded to one 16-byte
// vector; FP64 ones stay at 24 bytes, for more ring slots.
template <typename T, int B>
constexpr unsigned kTiXw = (B == 3 && sizeof(T) == 4) ? 4 : B;

// Record of one group: codes [G][S][msc], then values in 16-byte chunks
// (chunk k of lane l at vo + (kLanes k + l) 16): the B values of slot 0, 1, ...
struct TileGeom {
  unsigned ms, msc, nch, vo, gbytes;
};

template <int B, int S>
inline TileGeom tile_geom(unsigned ms, unsigned vs) {
  using L = TileLanes<B, S>;
  TileGeom g;
  g.ms = ms;
  g.msc = (ms + 3u) & ~3u;
  g.nch = (B * ms * vs + 15u) / 16u;
  g.vo = 4u * L::kG * S * g.msc;
  g.gbytes = g.vo + g.nch * L::kLanes * 16u;
  return g;
}

// A step's record: its groups, then its row list; the slot keeps the fetched
// rows behind it, at area_off.
struct TileArgs {
  unsigned ntiles, zero, gbytes, nslots, slot_bytes, area_off, ring_off;
  const uint4 *tiles, *steps;
  const unsigned char *bytes;
  unsigned *ctr;
  int *err;
  unsigned long long timeout_ns;
  const int *skip;
};

// One row in shared memory: B values, read as one vector.
template <typename T, int B>
__device__ __forceinline__ void tile_row(const unsigned char *p, T x[B]) {
  if constexpr (B == 3 && sizeof(T) == 4) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    x[0] = v.x;
    x[1] = v.y;
    x[2] = v.z;
  } else if constexpr (B == 3) {
#pragma unroll
    for (int k = 0; k < 3; ++k) x[k] = reinterpret_cast<const double *>(p)[k];
  } else if constexpr (B == 2 && sizeof(T) == 4) {
    const float2 v = *reinterpret_cast<const float2 *>(p);
    x[0] = v.x;
    x[1] = v.y;
  } else if constexpr (B == 2) {
    const double2 v = *reinterpret_cast<const double2 *>(p);
    x[0] = v.x;
    x[1] = v.y;
  } else {
    x[0] = *reinterpret_cast<const T *>(p);
  }
}

// tiles[t] = {first step, steps, offset and length of its records / 16};
// steps[s] = {offset and length of its record / 16, groups | own rows << 8 |
// list rows << 16, local index of its first row}; a step's list: its own rows,
// then the rows of other tiles it reads. ctr[0] hands out the tiles in order,
// so that a tile only waits for tiles that CTAs already running have (no CTA
// has to be resident at another's start); ctr[1] counts finished CTAs (the last
// one resets both).
template <typename T, int B, int S, int NW, int HW, int MS, bool FWD>
__global__ void __launch_bounds__(32 * (NW + HW + 1), 1)
    k_sweep_tiles(const TileArgs A, const T *__restrict__ in, T *out) {
  using L = TileLanes<B, S>;
  extern __shared__ __align__(128) unsigned char ti_smem[];
  pdl_wait();
  if (A.skip && *A.skip) return;
  uint64_t *full = reinterpret_cast<uint64_t *>(ti_smem);
  uint4 *smeta = reinterpret_cast<uint4 *>(ti_smem + 256);  // {groups | own << 8 | list << 16, local base, -, tile}
  volatile int *sstop = reinterpret_cast<volatile int *>(ti_smem + 512);  // per slot: its fetch warp gave up
  volatile unsigned *sdone = reinterpret_cast<volatile unsigned *>(ti_smem + 576);  // steps the consumers are done with
  unsigned char *xs = ti_smem + kTiXsOff;
  unsigned char *ring = ti_smem + A.ring_off;
  constexpr unsigned kXw = kTiXw<T, B>, kRow = kXw * sizeof(T);  // values, bytes of a row in shared memory
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;

  if (threadIdx.x == 0) {
    for (unsigned k = 0; k < A.nslots; ++k) {
      mbar_init(&full[k], 1);
      sstop[k] = 0;
    }
    *sdone = 0;
    mbar_fence_init();
  }
  if (threadIdx.x < kXw) reinterpret_cast<T *>(xs + (size_t)A.zero * kRow)[threadIdx.x] = T(0);
  __syncthreads();

  if (warp == NW + HW) {
    // ---- producer (one lane): walks the CTA's tiles and copies their steps,
    // one bulk copy each, as soon as the consumers have left a slot (sdone).
    // Descriptors are read kTiDesc steps ahead, each into registers of its own
    // (moving one on would wait for its load). The CTA's next tile is taken a
    // few steps before the current one ends (so tiles go to CTAs in the order
    // CTAs become free). Records are prefetched into L2 kTiAhead bytes before
    // they are copied, so that the ring only has to cover L2's latency. The end
    // is announced in HW slots, so that every fetch warp meets it. (A whole-warp
    // producer with an mbarrier wait per slot took 800 cycles a step and
    // bounded FP32 sweeps.)
    if (lane != 0) return;
    unsigned issued = 0, slot = 0, done = 0;
    auto room = [&]() -> bool {  // a free slot, bounded
      if (issued - done < A.nslots) return true;
      unsigned long long t0 = 0;
      unsigned spins = 0;
      for (;;) {
        done = *sdone;
        if ((int)(issued - done) < (int)A.nslots) break;
        if ((++spins & 255u) == 0) {
          const unsigned long long now = globaltimer_ns();
          if (t0 == 0) t0 = now;
          if (now - t0 > A.timeout_ns) {
            atomicCAS(A.err, 0, DFM2G_ERR_WAIT_TIMEOUT);
            return false;  // the other warps stop on their own bounded waits
          }
        }
      }
      __threadfence_block();
      return true;
    };
    auto next_slot = [&]() {
      ++issued;
      if (++slot == A.nslots) slot = 0;
    };
    auto mark = [&](const uint4 &m) -> bool {  // a slot without a record
      if (!room()) return false;
      smeta[slot] = m;
      mbar_arrive(&full[slot]);
      next_slot();
      return true;
    };
    // prefetch of 16-byte units [pf, to), at most `most` bytes
    auto prefetch = [&](unsigned &pf, unsigned to, unsigned most) {
      const unsigned n = min(to - pf, most / 16u);
      if (n) bulk_prefetch_l2(A.bytes + (size_t)pf * 16u, n * 16u);
      pf += n;
    };
    unsigned cur = atomicAdd(A.ctr, 1u);
    bool ok = true;
    const bool any = cur < A.ntiles;  // false: other CTAs took every tile before this one started
    uint4 td = A.tiles[any ? cur : 0u];
    unsigned pf = td.z;
    if (any) prefetch(pf, td.z + td.w, kTiAhead);
    while (ok && any) {
      const uint4 *sp = A.steps + td.x;
      uint4 d[kTiDesc], ntd = td;
#pragma unroll
      for (unsigned k = 0; k < kTiDesc; ++k) d[k] = k < td.y ? sp[k] : make_uint4(0u, 0u, 0u, 0u);
      unsigned tok = 0, next = kTiEnd, npf = 0;
      bool taken = false;
      for (unsigned c0 = 0; c0 < td.y && ok; c0 += kTiDesc) {
#pragma unroll
        for (unsigned k = 0; k < kTiDesc; ++k) {
          const unsigned cs = c0 + k;
          if (cs >= td.y || !ok) continue;
          if (!taken && cs + kTiGrabLead >= td.y) {
            tok = atomicAdd(A.ctr, 1u);
            taken = true;
          }
          if (next == kTiEnd && taken && (cs + kTiGrabLead / 2 >= td.y || cs + 1 == td.y)) {
            next = tok;
            if (next < A.ntiles) {
              ntd = A.tiles[next];
              npf = ntd.z;
              prefetch(npf, ntd.z + ntd.w, kTiAhead);
            }
          }
          ok = room();
          if (!ok) continue;
          const unsigned len = d[k].y * 16u;
          smeta[slot] = make_uint4(d[k].z, d[k].w, 0u, cur);
          mbar_arrive_expect_tx(&full[slot], len);
          tma_load_1d(ring + (size_t)slot * A.slot_bytes, A.bytes + (size_t)d[k].x * 16u, len, &full[slot]);
          next_slot();
          prefetch(pf, td.z + td.w, len);
          if (cs + kTiDesc < td.y) d[k] = sp[cs + kTiDesc];
        }
      }
      if (!ok || next >= A.ntiles) break;
      cur = next;
      td = ntd;
      pf = npf;
    }
    for (unsigned e = 0; e < HW && ok; ++e) ok = mark(make_uint4(e, 0u, 0u, kTiEnd));
    // wait (bounded) for the bulk copies of the last slots before leaving
    const unsigned lo = issued > A.nslots ? issued - A.nslots : 0u;
    for (unsigned i = lo; i < issued; ++i) mbar_wait_bounded(&full[i % A.nslots], (i / A.nslots) & 1u, A.timeout_ns);
    __threadfence();
    if (atomicAdd(A.ctr + 1, 1u) == gridDim.x - 1u) {
      atomicExch(A.ctr, 0u);
      atomicExch(A.ctr + 1, 0u);
    }
    return;
  }

  // Barrier at the end of step s: the consumers, the fetch warp of step s + 1
  // (its operands are in the slot) and that of step s + 2 (its record has
  // landed). Its id goes by the slot of step s + 2: a fetch warp ahead by up to
  // a ring meets no earlier step's barrier. The record of step 0 has a barrier
  // of its own (kFirst, the consumers and one fetch warp).
  constexpr int kMeet = 32 * (NW + 2), kFirst = 15;
  static_assert(kTiMaxSlots < kFirst, "barrier ids");

  if (warp >= NW) {
    // ---- fetch warps: lane kB lr + c reads component c of every kRp-th row of
    // the list, from the lr-th on (own rows: all of them in flight at once;
    // rows of other tiles: kFh per lane at a time)
    constexpr unsigned kRp = 32 / B, kFh = 4;
    constexpr unsigned kFo = (NW * L::kG + kRp - 1) / kRp;
    const unsigned lr = lane / B, c = lane - lr * B;
    const bool on = lr < kRp;
    unsigned slot = warp - NW, par = 0;
    bool first = warp == NW;
    // the record of the step in `slot` has landed (or its warp gives up)
    auto arrive_record = [&]() {
      if (first)
        asm volatile("bar.arrive %0, %1;" ::"n"(kFirst), "n"(32 * (NW + 1)) : "memory");
      else
        asm volatile("bar.arrive %0, %1;" ::"r"(slot + 1u), "n"(kMeet) : "memory");
      first = false;
    };
    for (;; slot += HW) {
      if (slot >= A.nslots) {
        slot -= A.nslots;
        par ^= 1u;
      }
      const bool landed = mbar_wait_bounded(&full[slot], par, A.timeout_ns);
      if (!__all_sync(0xffffffffu, landed)) {
        if (lane == 0) {
          atomicCAS(A.err, 0, DFM2G_ERR_WAIT_TIMEOUT);
          sstop[slot] = 1;
        }
        __syncwarp();
        arrive_record();
        return;
      }
      const uint4 meta = smeta[slot];
      if (meta.w == kTiEnd) {
        if (meta.x == 0) arrive_record();
        return;
      }
      arrive_record();
      unsigned char *sp = ring + (size_t)slot * A.slot_bytes;
      const unsigned *list = reinterpret_cast<const unsigned *>(sp + (meta.x & 0xFFu) * A.gbytes);
      const unsigned own = (meta.x >> 8) & 0xFFu, rows = meta.x >> 16;
      T *area = reinterpret_cast<T *>(sp + A.area_off + lr * kRow) + c;
      T rhs[kFo];
#pragma unroll
      for (unsigned k = 0; k < kFo; ++k) {
        const unsigned r = lr + kRp * k;
        rhs[k] = T(0);
        if (on && r < own) rhs[k] = in[(size_t)list[r] * B + c];
      }
      for (unsigned r0 = own + lr; on && r0 < rows; r0 += kRp * kFh) {
        T v[kFh];
        const T *src[kFh];
#pragma unroll
        for (unsigned k = 0; k < kFh; ++k) {
          const unsigned r = r0 + kRp * k;
          src[k] = (const T *)out + (size_t)list[r < rows ? r : r0] * B + c;
        }
#pragma unroll
        for (unsigned k = 0; k < kFh; ++k) v[k] = ld_relaxed(src[k]);
        auto pending = [&]() {
          bool p = false;
#pragma unroll
          for (unsigned k = 0; k < kFh; ++k) p |= is_pending(v[k]);
          return p;
        };
        if (pending()) {
          // not written yet (this tile runs close behind another): polled in L2
          // (all pending values at each poll: polling one a lane and reading the
          // others after it, or two staggered reads of each, measured 0-5% slower)
          unsigned long long t0 = 0;
          unsigned spins = 0;
          do {
#pragma unroll
            for (unsigned k = 0; k < kFh; ++k)
              if (is_pending(v[k])) v[k] = ld_relaxed(src[k]);
            if ((++spins & 63u) == 0) {
              const unsigned long long now = globaltimer_ns();
              if (t0 == 0) t0 = now;
              if (ld_relaxed(A.err) != 0 || now - t0 > A.timeout_ns) {
                atomicCAS(A.err, 0, DFM2G_ERR_WAIT_TIMEOUT);
                break;  // the values stay pending markers (NaN); the call reports the error
              }
            }
          } while (pending());
        }
        T *to = area + (size_t)(r0 - lr) * kXw;
#pragma unroll
        for (unsigned k = 0; k < kFh; ++k)
          if (r0 + kRp * k < rows) to[kRp * k * kXw] = v[k];
      }
#pragma unroll
      for (unsigned k = 0; k < kFo; ++k)
        if (on && lr + kRp * k < own) area[kRp * k * kXw] = settled(rhs[k]);
      __threadfence_block();
      __syncwarp();
      asm volatile("bar.arrive %0, %1;" ::"r"(slot + 1u == A.nslots ? 1u : slot + 2u), "n"(kMeet) : "memory");
    }
  }

  // ---- consumers
  const bool lane_ok = lane < L::kLanes;
  const unsigned q = lane_ok ? lane / L::kLpr : 0u, sub = lane_ok ? lane % L::kLpr : 0u;
  const unsigned h = sub / B, a = sub - h * B;
  const unsigned half0 = q * L::kLpr + h * B;  // first lane of this row's half
  constexpr unsigned kPer = 16u / sizeof(T);
  constexpr unsigned kNv = B * MS;
  constexpr unsigned kMsc = (MS + 3) / 4 * 4;
  constexpr unsigned kVo = 4u * L::kG * S * kMsc;

  // FP32: one chain of products per component of the operands, added at the
  // end; FP64: one chain, no extra additions on its narrow pipe
  constexpr int kAcc = sizeof(T) == 4 ? B : 1;
  constexpr bool kLast = FWD && sizeof(T) == 4;  // D^-1 applied to the finished sum: slot MS - 1 of half S - 1
  constexpr unsigned kOut = kLast ? S - 1 : 0;   // the half that holds the result
  constexpr unsigned kDeps = kLast ? MS - 1 : MS;
  const unsigned pos = warp * L::kG + q;  // the lane's row among the step's

  // A warp without a group in a step works on group 0 and stores nothing: the
  // step stays one straight piece of code, the next step's loads between its
  // products (skipping such warps' work measured 2-8% slower in FP32).
  struct Step {
    unsigned row, local, area;
    unsigned at[kMsc];  // operand offsets: codes until place(), then from ti_smem
    T v[(kNv + kPer - 1) / kPer * kPer];
  };
  // codes and values of the step in `slot`; false: the CTA is done
  auto load = [&](Step &N, unsigned slot, const uint4 meta, int stop) -> bool {
    const unsigned ng = meta.x & 0xFFu;
    const bool more = meta.w != kTiEnd && stop == 0;
    const unsigned so = slot * A.slot_bytes;
    N.area = A.ring_off + so + A.area_off;
    const unsigned char *gp = ring + so + (warp < ng ? warp * A.gbytes : 0u);
    const uint4 *cw = reinterpret_cast<const uint4 *>(gp + (q * S + h) * kMsc * 4u);
#pragma unroll
    for (unsigned k = 0; k < kMsc / 4; ++k) {
      const uint4 c = cw[k];
      N.at[4 * k + 0] = c.x;
      N.at[4 * k + 1] = c.y;
      N.at[4 * k + 2] = c.z;
      N.at[4 * k + 3] = c.w;
    }
    const bool valid = lane_ok && pos < ((meta.x >> 8) & 0xFFu);
    const unsigned row = reinterpret_cast<const unsigned *>(ring + so + ng * A.gbytes)[valid ? pos : 0u];
    N.row = valid ? row : ~0u;
    N.local = meta.y + pos;
    const unsigned char *vp = gp + kVo + (lane_ok ? lane : 0u) * 16u;
#pragma unroll
    for (unsigned k = 0; k < (kNv + kPer - 1) / kPer; ++k) {
      if constexpr (sizeof(T) == 4) {
        const float4 c = *reinterpret_cast<const float4 *>(vp + k * (L::kLanes * 16u));
        N.v[4 * k + 0] = c.x;
        N.v[4 * k + 1] = c.y;
        N.v[4 * k + 2] = c.z;
        N.v[4 * k + 3] = c.w;
      } else {
        const double2 c = *reinterpret_cast<const double2 *>(vp + k * (L::kLanes * 16u));
        N.v[2 * k + 0] = c.x;
        N.v[2 * k + 1] = c.y;
      }
    }
    return more;
  };
  // codes to offsets: the rows' own are offsets already, kTiSlot marks one in the slot's fetched rows
  auto place = [&](Step &N) {
    const unsigned base = N.area - kTiSlot;
#pragma unroll
    for (unsigned j = 0; j < MS; ++j)
      if ((int)N.at[j] < 0) N.at[j] += base;
  };
  unsigned s0 = 0, done = 0;
  // step C (in slot s0) finished, step N loaded; false: the CTA is done
  auto step = [&](Step &C, Step &N) -> bool {
    const unsigned s1 = s0 + 1u == A.nslots ? 0u : s0 + 1u;
    asm volatile("bar.sync %0, %1;" ::"r"(s1 + 1u), "n"(kMeet) : "memory");
    // every consumer is done with the steps before this one (the barrier orders
    // their reads before this store; a fence would cost 120 cycles)
    if (threadIdx.x == 0) *sdone = done;
    ++done;
    // the next step's descriptor first: shared memory answers in order
    const uint4 meta = smeta[s1];
    const int stop = sstop[s1];
    T x[MS * B], c = T(0);
#pragma unroll
    for (unsigned j = 0; j < MS; ++j)  // (the slot of D^-1 holds a dependency on the other half)
      if (j < kDeps || S > 1) tile_row<T, B>(ti_smem + C.at[j], x + j * B);
    if constexpr (!FWD || kLast) c = reinterpret_cast<const T *>(ti_smem + C.area + (C.row != ~0u ? pos : 0u) * kRow)[a];
    const bool more = load(N, s1, meta, stop);
    T acc[kAcc];
#pragma unroll
    for (unsigned k = 0; k < kAcc; ++k) acc[k] = T(0);
#pragma unroll
    for (unsigned j = 0; j < MS; ++j) {
      if (j < kDeps || (S > 1 && h != S - 1)) {
#pragma unroll
        for (unsigned k = 0; k < B; ++k) acc[k % kAcc] += C.v[j * B + k] * x[j * B + k];
      }
    }
    T z = acc[0];
#pragma unroll
    for (unsigned k = 1; k < kAcc; ++k) z += acc[k];
    if constexpr (S == 2) z += __shfl_sync(0xffffffffu, z, lane_ok ? (h == 0 ? lane + B : lane - B) : lane);
    // the finished sum is subtracted: started from the right-hand side, the
    // chain would round at its magnitude in every product (forward FP32 1.2e-7
    // against 8.2e-8, backward FP64 1.8e-16 against 0.9e-16)
    if constexpr (sizeof(T) == 4 || !FWD)
      z = c - z;
    else
      z = -z;
    if constexpr (kLast) {
      T t = T(0);
#pragma unroll
      for (unsigned k = 0; k < B; ++k)
        t += C.v[(MS - 1) * B + k] * (B == 1 ? z : __shfl_sync(0xffffffffu, z, half0 + k));
      z = t;
    }
    if (C.row != ~0u && h == kOut) {
      reinterpret_cast<T *>(xs + (size_t)C.local * kRow)[a] = z;
      st_relaxed(out + (size_t)C.row * B + a, z);
    }
    if (!more) {
      // the end markers need this slot too (they touch only its descriptor)
      if (threadIdx.x == 0) *sdone = done - 1u + A.nslots;
      return false;
    }
    place(N);
    s0 = s1;
    return true;
  };
  Step P0, P1;
  asm volatile("bar.sync %0, %1;" ::"n"(kFirst), "n"(32 * (NW + 1)) : "memory");
  if (!load(P0, 0, smeta[0], sstop[0])) return;
  place(P0);
  while (step(P0, P1) && step(P1, P0)) {
  }
}

}  // namespace dfm2g
