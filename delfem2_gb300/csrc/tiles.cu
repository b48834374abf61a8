// Tile schedule of the triangular sweeps (DFM2G_SWEEP_TILES; DFM2G_SWEEP_CHAINS
// for patterns whose rows fit its records), 1x1, 2x2 and 3x3 blocks, FP32 and
// FP64: partition, records and launch of the kernel of tile_kernel.cuh.
//
// The rows of one sweep direction are partitioned into tiles: bundles of
// segments of dependency chains (strands), grown from a seed row, a row
// joining the tile only once every row it depends on is in an earlier tile or
// already in this one. Seeds are taken in the sweep's (level, row) order, so
// the tiles are numbered in a dependency order that follows the wavefront.
// Inside a tile the rows are grouped by their local level (1 + the highest
// local level of the rows of the same tile they depend on): the tile's steps,
// at most one row per segment each. On a structured mesh in its natural order
// the tiles are columns of the grid (bundles of z lines of up to 65 rows on the
// voxel meshes), and a dependency path crosses a tile boundary once per tile
// instead of once per row or pencil of rows.
//
// Progress: tiles are handed out in increasing number from a counter, to CTAs
// that are running, and every dependency of a tile's row lies in a
// lower-numbered tile or in an earlier step of the same tile. The
// lowest-numbered unfinished tile is the current tile of some running CTA (a
// CTA's next tile is numbered above its current one), and all its outside
// dependencies are finished, so the sweep cannot deadlock, wherever and whenever
// the CTAs are placed. Every wait is bounded (DFM2G_ERR_WAIT_TIMEOUT); a CTA that
// stops early first waits (bounded) for the copies it issued.
#include <algorithm>
#include <atomic>
#include <functional>
#include <mutex>
#include <queue>
#include <thread>
#include <vector>

#include "common.cuh"
#include "tile_kernel.cuh"

namespace dfm2g {

// The tile partition of one direction (host only). `order` is the sweep's
// (level, row) order.
//
// Strands first: a row continues the strand of the dependency nearest to it
// in row number when it is also that row's successor nearest to it (on a grid
// numbered z fastest: its z neighbour, so the strands are the grid's z lines);
// any other row starts a strand. Each strand is cut into segments of nearly equal
// length, at most max_rows / max_segs rows. The rows of a segment depend on
// one another in a chain, so a segment has at most one row on each local
// level of a tile.
//
// Then the tiles: each grows from the first unassigned row of the level order
// (its seed: every row it depends on has a lower level, so it is assigned) by
// offers (layer, rank in the level order), smallest first. A row's successors
// are offered at the row's layer when they are in its segment, one layer
// further when they are in another strand, and after every other offer within
// reach when they start the next segment of its strand, so a tile takes the
// seed's segment, then the segments next to it at the same depth, and so on:
// on the voxel grids, square columns of z-line segments. A row joins once every
// row it depends on is assigned (to an earlier
// tile or this one), as long as the tile has fewer than max_rows rows, its
// segment is in the tile or the tile has fewer than max_segs segments, and
// its local level has fewer than max_width rows. The tiles are numbered along
// the wavefront. Outputs per row: its tile and local level; m = the most
// dependencies of a row. give_up > 0: *gave_up tells whether, once a sixteenth
// of the rows was assigned, they were ever in tiles of fewer than give_up rows on
// average; without force the partition stops there (ntiles = 0).
constexpr unsigned kTiSegFar = 1u << 20;  // layer step to the next segment of the same strand

void tile_partition(unsigned n, const unsigned *rs, const unsigned *dia, const unsigned *col, const unsigned *order,
                    bool fwd, unsigned max_rows, unsigned max_segs, unsigned max_width,
                    std::vector<unsigned> &tile_of, std::vector<unsigned> &lev, unsigned &ntiles, unsigned &m,
                    unsigned give_up, bool force, bool *gave_up) {
  const unsigned none = ~0u;
  if (gave_up) *gave_up = false;
  tile_of.assign(n, none);
  lev.assign(n, 0u);
  m = 0;
  auto dep_range = [&](unsigned i, unsigned &s0, unsigned &s1) {
    s0 = fwd ? rs[i] : dia[i];
    s1 = fwd ? dia[i] : rs[i + 1];
  };
  std::vector<unsigned> pos(n);  // rank in the level order
  for (unsigned k = 0; k < n; ++k) pos[order[k]] = k;
  // successors: rows that depend on each row
  std::vector<unsigned> sptr(n + 1, 0u), succ;
  for (unsigned i = 0; i < n; ++i) {
    unsigned s0, s1;
    dep_range(i, s0, s1);
    m = std::max(m, s1 - s0);
    for (unsigned s = s0; s < s1; ++s) sptr[col[s] + 1]++;
  }
  for (unsigned i = 0; i < n; ++i) sptr[i + 1] += sptr[i];
  succ.resize(sptr[n]);
  {
    std::vector<unsigned> fill(sptr.begin(), sptr.end() - 1);
    for (unsigned i = 0; i < n; ++i) {
      unsigned s0, s1;
      dep_range(i, s0, s1);
      for (unsigned s = s0; s < s1; ++s) succ[fill[col[s]]++] = i;
    }
  }
  // strands: r continues the strand of d when d is the dependency of r
  // nearest to it in row number and r the successor of d nearest to d (ties:
  // the earlier in the level order), so a row cannot take another's strand
  std::vector<unsigned> next(n, none), prev(n, none), near_succ(n, none);
  auto nearer = [&](unsigned r, unsigned cand, unsigned cur) {  // cand nearer to r than cur
    if (cur == none) return true;
    const unsigned dc = cand > r ? cand - r : r - cand, du = cur > r ? cur - r : r - cur;
    return dc < du || (dc == du && pos[cand] < pos[cur]);
  };
  for (unsigned d = 0; d < n; ++d)
    for (unsigned k = sptr[d]; k < sptr[d + 1]; ++k)
      if (nearer(d, succ[k], near_succ[d])) near_succ[d] = succ[k];
  for (unsigned r = 0; r < n; ++r) {
    unsigned s0, s1;
    dep_range(r, s0, s1);
    unsigned best = none;
    for (unsigned s = s0; s < s1; ++s)
      if (nearer(r, col[s], best)) best = col[s];
    if (best != none && near_succ[best] == r) {
      next[best] = r;
      prev[r] = best;
    }
  }
  // segments: strands cut into ceil(len / seg_max) pieces of nearly equal length
  const unsigned seg_max = std::max(1u, max_rows / std::max(1u, max_segs));
  std::vector<unsigned> seg_of(n, none);
  unsigned nseg_total = 0;
  for (unsigned r = 0; r < n; ++r) {
    if (prev[r] != none) continue;
    unsigned len = 0;
    for (unsigned u = r; u != none; u = next[u]) ++len;
    const unsigned pieces = (len + seg_max - 1u) / seg_max;
    unsigned k = 0;
    for (unsigned u = r; u != none; u = next[u], ++k) seg_of[u] = nseg_total + (unsigned)((uint64_t)k * pieces / len);
    nseg_total += pieces;
  }
  // offers (layer, rank), smallest first; layer_of[r]: the lowest layer r was offered at in this tile.
  // A row is offered once, when its last unassigned dependency joins the tile (unassigned[r] reaches 0).
  using Offer = std::pair<unsigned, unsigned>;
  std::priority_queue<Offer, std::vector<Offer>, std::greater<Offer>> heap;
  std::vector<unsigned> layer_of(n, none), offered;  // offered: rows whose layer_of is set in this tile
  std::vector<unsigned> width, seg_tile(nseg_total, none), unassigned(n);
  for (unsigned i = 0; i < n; ++i) {
    unsigned s0, s1;
    dep_range(i, s0, s1);
    unassigned[i] = s1 - s0;
  }
  unsigned cursor = 0, t = 0;
  size_t assigned = 0;
  for (;;) {
    while (cursor < n && tile_of[order[cursor]] != none) ++cursor;
    if (cursor >= n) break;
    if (give_up && assigned >= n / 16u && assigned < (size_t)give_up * t) {
      *gave_up = true;
      if (!force) {
        ntiles = 0;
        return;
      }
    }
    const unsigned seed = order[cursor];
    for (unsigned r : offered) layer_of[r] = none;
    offered.clear();
    while (!heap.empty()) heap.pop();
    heap.push(Offer(0u, pos[seed]));
    layer_of[seed] = 0;
    offered.push_back(seed);
    width.assign(max_rows + 1u, 0u);
    unsigned count = 0, nseg = 0;
    while (!heap.empty() && count < max_rows) {
      const Offer o = heap.top();
      heap.pop();
      const unsigned r = order[o.second];
      if (tile_of[r] != none) continue;
      const bool new_seg = seg_tile[seg_of[r]] != t;
      if (new_seg && nseg >= max_segs) continue;
      unsigned s0, s1;
      dep_range(r, s0, s1);
      unsigned lv = 0;  // every dependency is assigned (the row was offered when the last one joined)
      for (unsigned s = s0; s < s1; ++s) {
        const unsigned d = col[s];
        if (tile_of[d] == t) lv = std::max(lv, lev[d] + 1u);
      }
      if (width[lv] >= max_width) continue;  // left to a later tile
      tile_of[r] = t;
      lev[r] = lv;
      width[lv]++;
      ++count;
      if (new_seg) {
        seg_tile[seg_of[r]] = t;
        ++nseg;
      }
      for (unsigned k = sptr[r]; k < sptr[r + 1]; ++k) {
        const unsigned u = succ[k];
        // same segment: same layer; another strand: one layer further; the
        // strand's next segment: after every other segment in reach
        const unsigned lay = o.first + (seg_of[u] == seg_of[r] ? 0u : prev[u] == r ? kTiSegFar : 1u);
        if (layer_of[u] == none) offered.push_back(u);
        layer_of[u] = std::min(layer_of[u], lay);
        if (--unassigned[u] == 0) heap.push(Offer(layer_of[u], pos[u]));
      }
    }
    assigned += count;
    ++t;
  }
  ntiles = t;
}

namespace {

constexpr size_t kTiSmemCap = 227u * 1024u;
// A slot's factor block: none, or D^-1.
constexpr unsigned kSrcNone = 0xFFFFFFFFu, kSrcDia = 0xFFFFFFFEu;
// Tiles of fewer rows than this on average are not swept unless asked for
// (DFM2G_SWEEP_TILES): rows numbered without order depend on 10 tiles at once,
// and a warp per chain with its thousands of polls in flight is ahead (64^3
// voxels, nodes permuted at random, 10 rows a tile: 230 us FP32 a sweep, 425
// over tiles; permuted within windows of 400, 20 rows: 1,640 against 950).
constexpr unsigned kTiLeastRows = 16;
constexpr unsigned kTiAutoDeps = 8;             // most dependency blocks of a row, and least
constexpr unsigned kTi64MinRows = 76u * 1024u;  // rows in FP64, of what tile_sweep calls full

inline unsigned pad128u(unsigned x) { return (x + 127u) & ~127u; }

// The host part of one direction's schedule (no CUDA calls, so both
// directions are built at once on two host threads).
struct TileHost {
  bool ok = false, thin = false;
  unsigned ntiles = 0, nsteps = 0, ms = 0, max_groups = 0, max_tile = 0, max_list = 0, max_record = 0;
  size_t ngroups = 0, stream16 = 0;
  std::vector<uint4> tiles, steps;
  std::vector<unsigned> codes, src, grow, lists, goff, loff;
};

struct TileShape {
  unsigned B, S, rows, segs, width;  // block size, lanes split, limits of a tile and of a step
  unsigned row_bytes, vs;            // bytes of a row in shared memory, of a value
  unsigned ms[4];                    // slots per lane the kernels are compiled for, ascending (0: none)
};

// Codes and slot sources from the partition. Slots of a row: its dependencies
// in column order, alternating over the S lane groups, and last (forward) D^-1
// in slot ms - 1 of the last lane group, its operand the row's right-hand side.
void tile_host_build(unsigned n, const std::vector<unsigned> &rs, const std::vector<unsigned> &col,
                     const std::vector<unsigned> &dia, const std::vector<unsigned> &order, bool fwd,
                     const TileShape &sh, bool force, TileHost &out) {
  out.ok = out.thin = false;
  std::vector<unsigned> tile_of, lev;
  unsigned ntiles = 0, m = 0;
  tile_partition(n, rs.data(), dia.data(), col.data(), order.data(), fwd, sh.rows, sh.segs, sh.width, tile_of, lev,
                 ntiles, m, kTiLeastRows / 3u, force, &out.thin);
  out.thin |= ntiles > 1 && n < (size_t)kTiLeastRows * ntiles;  // the pattern's, whether asked for or not
  if (out.thin && !force) return;
  const unsigned S = sh.S, G = 32u / (sh.B * S);
  const unsigned need = std::max(1u, (m + (fwd ? 1u : 0u) + S - 1u) / S);
  unsigned ms = 0;
  for (unsigned c : sh.ms)
    if (ms == 0 && c >= need) ms = c;
  if (ms == 0) return;  // rows too long for the lanes' registers
  const unsigned msc = (ms + 3u) & ~3u;
  const unsigned words = G * S * msc, sw = G * S * ms;
  // rows of each tile by (local level, level order)
  std::vector<unsigned> tstart(ntiles + 1, 0u), trows(n);
  for (unsigned i = 0; i < n; ++i) tstart[tile_of[i] + 1]++;
  for (unsigned t = 0; t < ntiles; ++t) tstart[t + 1] += tstart[t];
  {
    std::vector<unsigned> fill(tstart.begin(), tstart.end() - 1);
    for (unsigned k = 0; k < n; ++k) trows[fill[tile_of[order[k]]]++] = order[k];
  }
  std::vector<unsigned> local(n);
  unsigned max_tile = 0;
  for (unsigned t = 0; t < ntiles; ++t) {
    unsigned *b = trows.data() + tstart[t], *e = trows.data() + tstart[t + 1];
    std::stable_sort(b, e, [&](unsigned x, unsigned y) { return lev[x] < lev[y]; });
    const unsigned nr = (unsigned)(e - b);
    max_tile = std::max(max_tile, nr);
    for (unsigned k = 0; k < nr; ++k) local[b[k]] = k;
  }
  const unsigned unused = kTiXsOff + max_tile * sh.row_bytes;  // the zero row
  std::vector<uint4> tiles(ntiles), steps;
  std::vector<unsigned> codes, src, grow, lists, goff, loff, hidx(n, ~0u);
  const size_t groups_guess = n / G + n / 16 + 1;
  codes.reserve(groups_guess * words);
  src.reserve(groups_guess * sw);
  grow.reserve(groups_guess * G);
  // a group's record in 16-byte units (tile_geom)
  const unsigned gb16 = words / 4u + (sh.B * ms * sh.vs + 15u) / 16u * (G * sh.B * S);
  size_t ngroups = 0, offset = 0;  // offset: of the next record in the stream, in 16-byte units
  unsigned max_groups = 0, max_list = 0, max_record = 0;
  for (unsigned t = 0; t < ntiles; ++t) {
    const unsigned *b = trows.data() + tstart[t];
    const unsigned nr = tstart[t + 1] - tstart[t];
    const unsigned first_step = (unsigned)steps.size();
    const size_t first_off = offset;
    unsigned k = 0;
    while (k < nr) {
      unsigned k1 = k;
      while (k1 < nr && lev[b[k1]] == lev[b[k]]) ++k1;
      const unsigned w = k1 - k, ng = (w + G - 1) / G;
      codes.resize((ngroups + ng) * words, unused);
      src.resize((ngroups + ng) * sw, kSrcNone);
      grow.resize((ngroups + ng) * G, ~0u);
      const size_t l0 = lists.size(), h0 = l0 + w;
      lists.insert(lists.end(), b + k, b + k1);  // the step's own rows, then the rows of other tiles
      for (unsigned u = k; u < k1; ++u) {
        const unsigned i = b[u], s0 = fwd ? rs[i] : dia[i], s1 = fwd ? dia[i] : rs[i + 1];
        for (unsigned s = s0; s < s1; ++s)
          if (tile_of[col[s]] != t && hidx[col[s]] == ~0u) {
            hidx[col[s]] = (unsigned)(lists.size() - h0);
            lists.push_back(col[s]);
          }
      }
      const unsigned hc = (unsigned)(lists.size() - h0);
      for (unsigned u = 0; u < w; ++u) {
        const unsigned i = b[k + u];
        const size_t g = ngroups + u / G;
        const unsigned q = u % G;
        unsigned *gp = codes.data() + g * words, *sp = src.data() + g * sw;
        grow[g * G + q] = i;
        const unsigned s0 = fwd ? rs[i] : dia[i], s1 = fwd ? dia[i] : rs[i + 1];
        for (unsigned s = s0; s < s1; ++s) {
          const unsigned j = (s - s0) / S, h = (s - s0) % S, d = col[s];
          gp[(q * S + h) * msc + j] =
              tile_of[d] == t ? kTiXsOff + local[d] * sh.row_bytes : kTiSlot + (w + hidx[d]) * sh.row_bytes;
          sp[(q * S + h) * ms + j] = s;
        }
        if (fwd) {
          gp[(q * S + S - 1u) * msc + ms - 1u] = kTiSlot + u * sh.row_bytes;
          sp[(q * S + S - 1u) * ms + ms - 1u] = kSrcDia;
        }
      }
      for (unsigned e = 0; e < hc; ++e) hidx[lists[h0 + e]] = ~0u;
      max_list = std::max(max_list, w + hc);
      while (lists.size() % 4u) lists.push_back(0u);
      const size_t lw = lists.size() - l0, rec = ng * (size_t)gb16 + lw / 4u;
      if (w + hc > 0xFFFFu || offset + rec >= 0xFFFFFFF0ull) return;  // descriptor fields
      for (unsigned g = 0; g < ng; ++g) goff.push_back((unsigned)(offset + g * (size_t)gb16));
      for (size_t e = 0; e < lw; e += 4) loff.push_back((unsigned)(offset + ng * (size_t)gb16 + e / 4u));
      steps.push_back(make_uint4((unsigned)offset, (unsigned)rec, ng | w << 8 | (w + hc) << 16, k));
      max_groups = std::max(max_groups, ng);
      max_record = std::max(max_record, (unsigned)rec);
      ngroups += ng;
      offset += rec;
      k = k1;
    }
    tiles[t] = make_uint4(first_step, (unsigned)steps.size() - first_step, (unsigned)first_off,
                          (unsigned)(offset - first_off));
  }
  out.ntiles = ntiles;
  out.nsteps = (unsigned)steps.size();
  out.ms = ms;
  out.max_groups = max_groups;
  out.max_tile = max_tile;
  out.max_list = max_list;
  out.max_record = max_record;
  out.stream16 = offset;
  out.ngroups = ngroups;
  out.tiles = std::move(tiles);
  out.steps = std::move(steps);
  out.codes = std::move(codes);
  out.src = std::move(src);
  out.grow = std::move(grow);
  out.lists = std::move(lists);
  out.goff = std::move(goff);
  out.loff = std::move(loff);
  out.ok = true;
}

unsigned tile_max_slots(const TileShape &sh) { return *std::max_element(sh.ms, sh.ms + 4); }

template <typename V>
int tile_to_host(std::vector<V> &h, const V *d, size_t n) {
  h.resize(n);
  if (n) DFM2G_CUDA(cudaMemcpy(h.data(), d, n * sizeof(V), cudaMemcpyDeviceToHost));
  return DFM2G_OK;
}

template <typename V>
int tile_to_dev(DevBuf<V> &d, const std::vector<V> &h) {
  DFM2G_TRY(d.resize(h.size()));
  if (!h.empty()) DFM2G_CUDA(cudaMemcpy(d.p, h.data(), h.size() * sizeof(V), cudaMemcpyHostToDevice));
  return DFM2G_OK;
}

int tile_upload(unsigned n, const TileHost &h, TileSched &ts) {
  ts.ok = false;
  ts.thin = h.thin;
  if (!h.ok) return DFM2G_OK;
  ts.ntiles = h.ntiles;
  ts.nsteps = h.nsteps;
  ts.rows_per_step = ts.nsteps ? (double)n / ts.nsteps : 0.0;
  ts.ngroups = h.ngroups;
  ts.max_groups = h.max_groups;
  ts.max_tile = h.max_tile;
  ts.max_list = h.max_list;
  ts.max_record = h.max_record;
  ts.stream16 = h.stream16;
  ts.ms = h.ms;
  DFM2G_TRY(tile_to_dev(ts.tiles, h.tiles));
  DFM2G_TRY(tile_to_dev(ts.steps, h.steps));
  DFM2G_TRY(tile_to_dev(ts.codes, h.codes));
  DFM2G_TRY(tile_to_dev(ts.src, h.src));
  DFM2G_TRY(tile_to_dev(ts.grow, h.grow));
  DFM2G_TRY(tile_to_dev(ts.lists, h.lists));
  DFM2G_TRY(tile_to_dev(ts.goff, h.goff));
  DFM2G_TRY(tile_to_dev(ts.loff, h.loff));
  DFM2G_TRY(ts.ctr.resize(2));
  DFM2G_CUDA(cudaMemset(ts.ctr.p, 0, 2 * sizeof(unsigned)));
  ts.ok = true;
  return DFM2G_OK;
}

// Builds the schedules of both directions of `pair` that are not built yet,
// their host parts on one thread each.
int tile_build(dfm2g_ilu_s *p, TileSched *pair, const TileShape &sh, bool force) {
  const unsigned n = p->nblk;
  bool need[2], any = false;
  for (int d = 0; d < 2; ++d) {
    need[d] = !pair[d].built || (force && pair[d].thin && !pair[d].forced);
    pair[d].built = true;
    if (need[d]) {
      pair[d].ok = pair[d].thin = false;
      pair[d].forced = force;
    }
    any |= need[d];
  }
  if (!any) return DFM2G_OK;
  // rows longer than the records hold need no partition
  for (int d = 0; d < 2; ++d)
    if ((d == 0 ? p->max_lower + 1u : p->max_upper) > tile_max_slots(sh) * sh.S) need[d] = false;
  if (!(need[0] || need[1]) || n >= kTiSlot) return DFM2G_OK;
  std::vector<unsigned> rs, col, dia, order[2];
  DFM2G_CUDA(cudaStreamSynchronize(stream()));
  DFM2G_TRY(tile_to_host(rs, p->row_start.p, (size_t)n + 1));
  DFM2G_TRY(tile_to_host(col, p->col.p, p->nnz));
  DFM2G_TRY(tile_to_host(dia, p->dia_ind.p, n));
  if (need[0]) DFM2G_TRY(tile_to_host(order[0], p->order_f.p, n));
  if (need[1]) DFM2G_TRY(tile_to_host(order[1], p->order_b.p, n));
  TileHost h[2];
  // an exception inside a worker (out of host memory) is caught there: it
  // leaves that schedule unusable and the call reports DFM2G_ERR_HOST
  std::atomic<bool> failed{false};
  std::vector<std::thread> workers;
  try {
    for (int d = 0; d < 2; ++d)
      if (need[d])
        workers.emplace_back([&, d]() {
          try {
            tile_host_build(n, rs, col, dia, order[d], d == 0, sh, force, h[d]);
          } catch (...) {
            h[d].ok = false;
            failed = true;
          }
        });
  } catch (...) {  // a thread that could not start: join the others before leaving
    for (std::thread &w : workers) w.join();
    throw;
  }
  for (std::thread &w : workers) w.join();
  if (failed) return fail(DFM2G_ERR_HOST, "tile schedule: out of host memory while partitioning");
  for (int d = 0; d < 2; ++d)
    if (need[d]) DFM2G_TRY(tile_upload(n, h[d], pair[d]));
  return DFM2G_OK;
}

// The parts of the records that do not depend on the values: each group's
// codes (cw 16-byte words at goff) and each step's row list (at loff).
__global__ void k_tile_lay(size_t ngroups, unsigned cw, const uint4 *__restrict__ codes,
                           const unsigned *__restrict__ goff, size_t nlist, const uint4 *__restrict__ lists,
                           const unsigned *__restrict__ loff, uint4 *__restrict__ stream16) {
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t nth = (size_t)gridDim.x * blockDim.x;
  for (size_t e = tid; e < ngroups * cw; e += nth) {
    const size_t g = e / cw;
    stream16[goff[g] + (e - g * cw)] = codes[e];
  }
  for (size_t e = tid; e < nlist; e += nth) stream16[loff[e]] = lists[e];
}

// The records' values of one value type from the FP64 factors, one 16-byte
// chunk per thread. Forward: D^-1 L and -D^-1 (FP64), L and D^-1 (FP32);
// backward: U'.
template <typename T, int B, int S, bool FWD>
__global__ void k_tile_fill(size_t ngroups, const double *__restrict__ vcrs, const double *__restrict__ vdia,
                            const unsigned *__restrict__ src, const unsigned *__restrict__ grow,
                            const unsigned *__restrict__ goff, TileGeom geo, uint4 *__restrict__ stream16) {
  using L = TileLanes<B, S>;
  constexpr unsigned PER = 16u / sizeof(T);
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t nth = (size_t)gridDim.x * blockDim.x;
  const unsigned per_group = geo.nch * L::kLanes;
  for (size_t e = tid; e < ngroups * per_group; e += nth) {
    const size_t g = e / per_group;
    const unsigned r = (unsigned)(e - g * per_group), k = r / L::kLanes, l = r - k * L::kLanes;
    const unsigned q = l / L::kLpr, sub = l - q * L::kLpr, h = sub / B, a = sub - h * B;
    const unsigned row = grow[g * L::kG + q];
    const unsigned *sp = src + (g * L::kG + q) * S * geo.ms + h * geo.ms;
    __align__(16) T v[PER];
#pragma unroll
    for (unsigned i = 0; i < PER; ++i) {
      const unsigned idx = k * PER + i, j = idx / B, c = idx - j * B;
      const unsigned s = j < geo.ms ? sp[j] : kSrcNone;
      double x = 0.0;
      if (row != ~0u && s != kSrcNone) {
        if constexpr (FWD) {
          const double *d = vdia + (size_t)row * (B * B) + a * B;
          if (s == kSrcDia) {
            x = sizeof(T) == 8 ? -d[c] : d[c];
          } else if (sizeof(T) == 4) {
            x = vcrs[(size_t)s * (B * B) + a * B + c];
          } else {
            const double *lb = vcrs + (size_t)s * (B * B) + c;
            x = d[0] * lb[0];
#pragma unroll
            for (int b = 1; b < B; ++b) x += d[b] * lb[b * B];
          }
        } else {
          x = vcrs[(size_t)s * (B * B) + a * B + c];
        }
      }
      v[i] = settled((T)x);  // as the right-hand side, in the kernel
    }
    stream16[(size_t)goff[g] + geo.vo / 16u + r] = *reinterpret_cast<const uint4 *>(v);
  }
}

// Lets `kernel` launch with `smem` bytes of dynamic shared memory. The
// attribute belongs to the kernel, not to a pattern, so it only ever grows
// (per kernel and device).
int tile_allow_smem(void *kernel, size_t smem) {
  struct Entry {
    void *kernel;
    int device;
    size_t smem;
  };
  static std::mutex mu;
  static std::vector<Entry> done;
  std::lock_guard<std::mutex> lock(mu);
  const int dev = ctx().device;
  for (auto &d : done) {
    if (d.kernel != kernel || d.device != dev) continue;
    if (d.smem >= smem) return DFM2G_OK;
    DFM2G_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    d.smem = smem;
    return DFM2G_OK;
  }
  DFM2G_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  done.push_back(Entry{kernel, dev, smem});
  return DFM2G_OK;
}

template <typename T, int B, int S, int NW, int HW, int MS>
void *tile_kernel(bool forward) {
  return forward ? (void *)k_sweep_tiles<T, B, S, NW, HW, MS, true>
                 : (void *)k_sweep_tiles<T, B, S, NW, HW, MS, false>;
}

template <typename T, int B, int S, int NW, int HW, int MSA, int MSB, int MSC, int MSD>
int tile_launch(dfm2g_ilu_s *p, TileSched &ts, bool forward, const T *in, T *out, size_t fill, const int *skip,
                unsigned long long timeout, bool *usable) {
  constexpr unsigned kRow = kTiXw<T, B> * (unsigned)sizeof(T);
  constexpr unsigned kThreads = 32 * (NW + HW + 1);
  const TileGeom g = tile_geom<B, S>(ts.ms, (unsigned)sizeof(T));
  TileArgs A{};
  A.ntiles = ts.ntiles;
  A.zero = ts.max_tile;
  A.gbytes = g.gbytes;
  A.area_off = ts.max_record * 16u;
  A.slot_bytes = pad128u(A.area_off + ts.max_list * kRow);
  A.ring_off = kTiXsOff + pad128u((ts.max_tile + 1u) * kRow);
  // a multiple of HW slots (each slot always the same fetch warp's), at least
  // four; half the shared memory where the tiles are many, so that two CTAs fit
  // an SM (FP64, 1,056 tiles: 430 us a sweep against 460; with fewer than four
  // per SM the longer ring is ahead, 297 tiles: 200 us against 225)
  const size_t cap = ts.ntiles >= 4u * (unsigned)ctx().num_sms ? kTiSmemCap / 2 - 1024 : kTiSmemCap;
  constexpr unsigned kLeast = HW >= 4 ? HW : 2 * HW;
  A.nslots = kTiMaxSlots / HW * HW;
  while (A.nslots > kLeast && A.ring_off + (size_t)A.nslots * A.slot_bytes > cap) A.nslots -= HW;
  const size_t smem = A.ring_off + (size_t)A.nslots * A.slot_bytes;
  if (smem > kTiSmemCap) return DFM2G_OK;  // long row lists (dense patterns): not even the shortest ring fits
  const unsigned fill_blocks = ctx().num_sms * 16;
  uint4 *stream16 = reinterpret_cast<uint4 *>(ts.bytes.p);
  if (!ts.bytes.p) {
    DFM2G_TRY(ts.bytes.resize(ts.stream16 * 16u));
    stream16 = reinterpret_cast<uint4 *>(ts.bytes.p);
    k_tile_lay<<<fill_blocks, 256, 0, stream()>>>(ts.ngroups, g.vo / 16u, reinterpret_cast<const uint4 *>(ts.codes.p),
                                                  ts.goff.p, ts.loff.n, reinterpret_cast<const uint4 *>(ts.lists.p),
                                                  ts.loff.p, stream16);
    DFM2G_LAUNCH_CHECK();
    note_launches(1);
    ts.ver = ~0u;
  }
  if (ts.ver != p->factor_version) {
    if (forward)
      k_tile_fill<T, B, S, true><<<fill_blocks, 256, 0, stream()>>>(ts.ngroups, p->vcrs.p, p->vdia.p, ts.src.p,
                                                                   ts.grow.p, ts.goff.p, g, stream16);
    else
      k_tile_fill<T, B, S, false><<<fill_blocks, 256, 0, stream()>>>(ts.ngroups, p->vcrs.p, p->vdia.p, ts.src.p,
                                                                    ts.grow.p, ts.goff.p, g, stream16);
    DFM2G_LAUNCH_CHECK();
    note_launches(1);
    ts.ver = p->factor_version;
  }
  void *kernel = ts.ms == MSA   ? tile_kernel<T, B, S, NW, HW, MSA>(forward)
                 : ts.ms == MSB ? tile_kernel<T, B, S, NW, HW, MSB>(forward)
                 : ts.ms == MSC ? tile_kernel<T, B, S, NW, HW, MSC>(forward)
                                : tile_kernel<T, B, S, NW, HW, MSD>(forward);
  DFM2G_TRY(tile_allow_smem(kernel, smem));
  if (ts.coop <= 0) {
    int per_sm = 0;
    DFM2G_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, smem));
    if (per_sm <= 0) return DFM2G_OK;
    ts.coop = per_sm * ctx().num_sms;
  }
  const unsigned blocks = std::min<unsigned>((unsigned)ts.coop, ts.ntiles);
  A.tiles = ts.tiles.p;
  A.steps = ts.steps.p;
  A.bytes = ts.bytes.p;
  A.ctr = ts.ctr.p;
  A.err = p->err.p;
  A.timeout_ns = timeout;
  A.skip = skip;
  void *args[] = {(void *)&A, (void *)&in, (void *)&out};
  DFM2G_TRY(fill_pending(out, fill));
  DFM2G_TRY(launch_after(kernel, blocks, kThreads, smem, args));
  note_launches(1);
  *usable = true;
  return DFM2G_OK;
}

// Prepares `pair` (both directions), sets `fill` bytes of `out` to the pending
// marker and sweeps; nothing is done (*usable
// stays false) when the pattern's rows are too long, or when !may_alloc and
// the records do not exist yet.
template <typename T, int B, int S, int NW, int HW, int MSA, int MSB, int MSC, int MSD>
int tile_run(dfm2g_ilu_s *p, TileSched *pair, const TileShape &sh, bool forward, const T *in, T *out, size_t fill,
             const int *skip, unsigned long long timeout, bool may_alloc, bool force, bool *usable) {
  TileSched &ts = pair[forward ? 0 : 1];
  if (!may_alloc && (!ts.built || !ts.ok || !ts.bytes.p)) return DFM2G_OK;
  if (!ts.built || (force && ts.thin && !ts.forced)) DFM2G_TRY(tile_build(p, pair, sh, force));
  if (!ts.ok || (ts.thin && !force)) return DFM2G_OK;
  return tile_launch<T, B, S, NW, HW, MSA, MSB, MSC, MSD>(p, ts, forward, in, out, fill, skip, timeout, usable);
}

// Shapes. The tiles are squares of z lines on the voxel grids (a row's offers
// spread over its neighbours' lines, diagonals included, so other segment
// counts grow ragged tiles: 16 lines swept 20% faster than 20). FP32 3x3: 6 x 6
// lines, three lanes a row. FP64 3x3: 4 x 4, six lanes a row on four warps (the
// step's 13 or 14 FP64 instructions per warp are its time, whatever the rows, so
// small tiles hop sooner: 65^3 nodes 200 us a sweep, 285 with 6 x 6 lines on
// eight warps). 1x1 and 2x2: two lane groups per row.
constexpr int kHw = 3, kHwNd = 4;  // fetch warps
constexpr TileShape kShape32{3, 1, 36 * 65, 36, 40, 16, 4, {7, 8, 14, 16}};
constexpr TileShape kShape64{3, 2, 16 * 65, 16, 20, 24, 8, {3, 4, 7, 8}};
template <typename T>
constexpr TileShape kShapeNd2{2, 2, 32 * 65, 32, 32, 2 * sizeof(T), sizeof(T), {4, 8, 0, 0}};
template <typename T>
constexpr TileShape kShapeNd1{1, 2, 64 * 65, 64, 64, sizeof(T), sizeof(T), {4, 8, 0, 0}};

}  // namespace

// The tile schedule of one direction (force: thin tiles too). *full tells whether its steps are full
// (at least half a step's segments on average, at most kTiAutoDeps
// dependencies a row, and in FP64 kTi64MinRows rows): the patterns that
// dfm2g_ilu_last_schedule calls tiles under DFM2G_SWEEP_AUTO. It is a name that
// callers know, and decides nothing: the same sweep over thinner patterns (cloth
// sheets, fill-in, 1x1 and 2x2 blocks, small FP64 systems) it calls chains, and
// dfm2g_ilu_last_kernel says what ran.
template <typename T>
int tile_sweep(dfm2g_ilu_s *p, bool forward, const T *in, T *out, size_t fill, const int *skip,
               unsigned long long timeout, bool may_alloc, bool force, bool *usable, bool *full) {
  constexpr bool f64 = sizeof(T) == 8;
  TileSched *pair = p->tiles[f64 ? 1 : 0];
  *usable = *full = false;
  if (p->ndim == 1)
    return tile_run<T, 1, 2, 4, kHwNd, 4, 8, 8, 8>(p, pair, kShapeNd1<T>, forward, in, out, fill, skip, timeout,
                                             may_alloc, force, usable);
  if (p->ndim == 2)
    return tile_run<T, 2, 2, 4, kHwNd, 4, 8, 8, 8>(p, pair, kShapeNd2<T>, forward, in, out, fill, skip, timeout,
                                             may_alloc, force, usable);
  constexpr TileShape sh = f64 ? kShape64 : kShape32;
  if constexpr (f64)
    DFM2G_TRY((tile_run<T, 3, 2, 4, kHw, 3, 4, 7, 8>(p, pair, sh, forward, in, out, fill, skip, timeout,
                                                     may_alloc, force, usable)));
  else
    DFM2G_TRY((tile_run<T, 3, 1, 4, kHw, 7, 8, 14, 16>(p, pair, sh, forward, in, out, fill, skip, timeout,
                                                       may_alloc, force, usable)));
  *full = *usable && (forward ? p->max_lower : p->max_upper) <= kTiAutoDeps &&
          2.0 * pair[forward ? 0 : 1].rows_per_step >= sh.segs && (!f64 || p->nblk >= kTi64MinRows);
  return DFM2G_OK;
}

template int tile_sweep<float>(dfm2g_ilu_s *, bool, const float *, float *, size_t, const int *, unsigned long long,
                               bool, bool, bool *, bool *);
template int tile_sweep<double>(dfm2g_ilu_s *, bool, const double *, double *, size_t, const int *, unsigned long long,
                                bool, bool, bool *, bool *);

// Drops the tiles and records (a new pattern); rebuilt on first use.
void tile_schedules_reset(dfm2g_ilu_s *p) {
  for (auto &pair : p->tiles)
    for (TileSched &ts : pair) {
      ts.built = ts.ok = ts.thin = ts.forced = false;
      ts.ntiles = ts.nsteps = ts.ms = ts.max_groups = ts.max_tile = ts.max_list = ts.max_record = 0;
      ts.rows_per_step = 0;
      ts.ngroups = ts.stream16 = 0;
      ts.ver = ~0u;
      ts.coop = 0;
      ts.tiles.release();
      ts.steps.release();
      ts.codes.release();
      ts.src.release();
      ts.grow.release();
      ts.lists.release();
      ts.goff.release();
      ts.loff.release();
      ts.bytes.release();
      ts.ctr.release();
    }
}

}  // namespace dfm2g

using namespace dfm2g;

extern "C" {

// Host-only: the tile partition the tile schedule uses. No device work.
int dfm2g_tile_partition(unsigned n, const unsigned *row_start, const unsigned *col, const unsigned *dia_ind,
                         const unsigned *order, int backward, unsigned max_rows, unsigned max_width,
                         unsigned *tile_of, unsigned *level, unsigned *ntiles, unsigned *max_deps) try {
  if (n && (!row_start || !col || !dia_ind || !order || !tile_of || !level))
    return fail(DFM2G_ERR_ARG, "tile_partition: null array");
  if (max_rows == 0 || max_width == 0) return fail(DFM2G_ERR_ARG, "tile_partition: zero tile size");
  std::vector<unsigned> t, lv;
  unsigned nt = 0, m = 0;
  tile_partition(n, row_start, dia_ind, col, order, backward == 0, max_rows, max_width, max_width, t, lv, nt, m, 0u,
                 false, nullptr);
  if (n) {
    std::copy(t.begin(), t.end(), tile_of);
    std::copy(lv.begin(), lv.end(), level);
  }
  if (ntiles) *ntiles = nt;
  if (max_deps) *max_deps = m;
  return DFM2G_OK;
} catch (...) {
  return host_failure();
}

}  // extern "C"
