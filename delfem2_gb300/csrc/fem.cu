// Linear tets on the device: atomic-free assembly of the elasticity K and b
// (3x3 blocks, per-tet Young's modulus), of the dynamic forms, of the scalar
// Poisson K and b (1x1 blocks), and the adjoint element term dL/dE.
//
// The matrix is gathered, not scattered: a thread owns a pair of blocks (i, j),
// (j, i) or a node and adds up the tets that touch it, in tet order, so each
// block is read and written once per assembly and the sums do not depend on
// the schedule. Lists made once per mesh: `elist` holds, edge by edge (the
// upper slots, compacted in `eslot`, offsets `eoff`), the codes 16 e + 4 a + b
// of the tets e with tet[e][a] = i, tet[e][b] = j; `nlist`, node by node
// (offsets `noff`), the codes with both nodes at i (a = b, and pairs of a tet
// that names a node twice). The tets' gradients and volume are made with them:
// geo[16 e + 4 k .. + 3) = dN_k, geo[16 e + 3] = vol.
//
// With moduli in a fixed ratio the tets' blocks come from one 3x3 sum,
// X = sum E vol dN_a dN_b^T: K_ij = lambda1 X + myu1 X^T + myu1 tr(X) I
// (AddEmat_LinearSolid3, include/delfem2/fem_solidlinear.cpp:55-79), 13 FP64
// operations per tet and edge where the element matrix takes 31; GB300's FP64
// pipe bounds the assembly, with the matrix read and written once next to it.
// 3.5M tets (96 x 95 x 64 voxels), K and b with a displacement: 1.95 ms (edges
// 0.95, nodes 0.66, stresses 0.34); scattering the element matrices colour by
// colour, four threads a tet and 33 launches, took 10.1 ms.
#include <algorithm>
#include <cstring>

#include "common.cuh"

namespace dfm2g {

constexpr unsigned kDiagSlot = 0xFFFFFFFFu;

// Volume and barycentric-coordinate gradients of a tet (the quantities of
// TetVolume3D / TetDlDx, include/delfem2/femutil.cpp:202-258): dN_k is the
// normal of the face opposite vertex k, scaled by 1/(6 vol), pointing to k.
__device__ __forceinline__ double tet_geometry(const double P[4][3], double dN[4][3]) {
  const double ax = P[1][0] - P[0][0], ay = P[1][1] - P[0][1], az = P[1][2] - P[0][2];
  const double bx = P[2][0] - P[0][0], by = P[2][1] - P[0][1], bz = P[2][2] - P[0][2];
  const double cx = P[3][0] - P[0][0], cy = P[3][1] - P[0][1], cz = P[3][2] - P[0][2];
  const double vol = (ax * (by * cz - cy * bz) - ay * (bx * cz - cx * bz) + az * (bx * cy - cx * by)) / 6.0;
  const double inv6v = 1.0 / (6.0 * vol);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double *a = P[(k + 1) & 3], *b = P[(k + 2) & 3], *c = P[(k + 3) & 3];
    const double ux = b[0] - a[0], uy = b[1] - a[1], uz = b[2] - a[2];
    const double wx = c[0] - a[0], wy = c[1] - a[1], wz = c[2] - a[2];
    const double s = ((k & 1) ? 1.0 : -1.0) * inv6v;
    dN[k][0] = s * (uy * wz - uz * wy);
    dN[k][1] = s * (uz * wx - ux * wz);
    dN[k][2] = s * (ux * wy - uy * wx);
  }
  return vol;
}

// ---- the gather lists ---------------------------------------------------------
__global__ void k_tet_geo(size_t ntet, const unsigned *__restrict__ tet, const double *__restrict__ xyz,
                          double *__restrict__ geo) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < ntet; e += (size_t)gridDim.x * blockDim.x) {
    double P[4][3], dN[4][3];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int d = 0; d < 3; ++d) P[k][d] = xyz[(size_t)tet[e * 4 + k] * 3 + d];
    const double vol = tet_geometry(P, dN);
    double2 *g = reinterpret_cast<double2 *>(geo + e * 16);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      g[2 * k] = make_double2(dN[k][0], dN[k][1]);
      g[2 * k + 1] = make_double2(dN[k][2], k == 0 ? vol : 0.0);
    }
  }
}

// Counts (fill = 0) or writes (fill = 1) the list entries of every (tet, a, b):
// edges by their upper slot, node entries by node.
__global__ void k_tet_lists(size_t ntet, const unsigned *__restrict__ tet, const unsigned *__restrict__ slot, int fill,
                            unsigned *edge_at, unsigned *node_at, unsigned *__restrict__ elist,
                            unsigned *__restrict__ nlist) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < ntet * 16;
       k += (size_t)gridDim.x * blockDim.x) {
    const size_t e = k >> 4;
    const unsigned i = tet[e * 4 + ((k >> 2) & 3)], j = tet[e * 4 + (k & 3)], s = slot[k];
    if (s == kDiagSlot) {
      const unsigned at = atomicAdd(node_at + i, 1u);
      if (fill) nlist[at] = (unsigned)k;
    } else if (i < j) {
      const unsigned at = atomicAdd(edge_at + s, 1u);
      if (fill) elist[at] = (unsigned)k;
    }
  }
}

// Exclusive scan of a[0, n) in tiles of kScanTile: tile sums, their scan by one
// block, and the tiles' own scans on top. `flag` scans (a[k] > 0) instead.
constexpr unsigned kScanTile = 2048;

__global__ void __launch_bounds__(256) k_scan_tile(const unsigned *__restrict__ a, unsigned n, int flag,
                                                   const unsigned *__restrict__ base, unsigned *__restrict__ out,
                                                   unsigned *__restrict__ sums) {
  __shared__ unsigned sh[8];
  const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const size_t k0 = (size_t)blockIdx.x * kScanTile + threadIdx.x * 8u;
  unsigned v[8], t = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const unsigned x = k0 + q < n ? a[k0 + q] : 0u;
    v[q] = t;
    t += flag ? (x > 0u) : x;
  }
  unsigned x = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (unsigned)o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  unsigned before = 0, all = 0;
  for (unsigned q = 0; q < 8; ++q) {
    if (q < w) before += sh[q];
    all += sh[q];
  }
  if (!out) {
    if (threadIdx.x == 0) sums[blockIdx.x] = all;
    return;
  }
  const unsigned off = base[blockIdx.x] + before + x - t;
#pragma unroll
  for (int q = 0; q < 8; ++q)
    if (k0 + q < n) out[k0 + q] = off + v[q];
}

__global__ void __launch_bounds__(1024) k_scan_sums(unsigned *sums, unsigned n, unsigned *total) {
  __shared__ unsigned sh[32];
  __shared__ unsigned carry;
  const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (unsigned k0 = 0; k0 < n; k0 += 1024) {
    const unsigned k = k0 + threadIdx.x, v = k < n ? sums[k] : 0u;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= (unsigned)o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    unsigned before = carry, all = 0;
    for (unsigned q = 0; q < 32; ++q) {
      if (q < w) before += sh[q];
      all += sh[q];
    }
    if (k < n) sums[k] = before + x - v;
    __syncthreads();
    if (threadIdx.x == 0) carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

// Edges with tets, compacted: eslot (their upper slot) and eoff (their first
// list entry); at[s]: the slot's first entry, rank[s]: its number among them.
__global__ void k_tet_edges_compact(unsigned nnz, const unsigned *__restrict__ count, const unsigned *__restrict__ at,
                                    const unsigned *__restrict__ rank, unsigned *__restrict__ eslot,
                                    unsigned *__restrict__ eoff) {
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < nnz; s += gridDim.x * blockDim.x) {
    if (count[s] == 0) continue;
    eslot[rank[s]] = s;
    eoff[rank[s]] = at[s];
  }
}

// Each list in ascending order (the fill's order is not deterministic).
__global__ void k_sort_lists(unsigned n, const unsigned *__restrict__ off, unsigned total, unsigned *list) {
  for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const unsigned b = off[k], e = k + 1 < n ? off[k + 1] : total;
    for (unsigned p = b + 1; p < e; ++p) {
      const unsigned v = list[p];
      unsigned q = p;
      while (q > b && list[q - 1] > v) {
        list[q] = list[q - 1];
        --q;
      }
      list[q] = v;
    }
  }
}

// ---- assembly -------------------------------------------------------------------
// Modes: kStatic: moduli E_e (lambda1, myu1), b_i += rho g vol/4 - (K u)_i
// (fem_solidlinear.h:192-237). kBEuler: MergeLinSys_SolidLinear_BEuler_MeshTet3D
// (fem_solidlinear.h:381-443): E = K + rho vol/(4 dt^2) I on the diagonal,
// b += (rho g vol/4 - K (u + dt v)) / dt. kWarp:
// MergeLinSys_SolidStiffwarp_BEuler_MeshTet3D (445-530): the same with
// K_ij <- R_i K_ij R_i^T and u_j + dt v_j <- P_j + u_j + dt v_j - R_i P_j (R_i =
// rot of node i, row-major). kNewmark:
// MergeLinSys_SolidLinear_NewmarkBeta_MeshTet3D (331-379, with
// EMat_SolidLinear_NewmarkBeta_MeshTet3D, fem_solidlinear.cpp:437-488, first
// iteration): M_ij = rho vol/20 (1 + [i == j]) I, E = M + beta dt^2 K,
// b += rho g vol/4 - K (u + dt v + dt^2/2 acc) - M acc.
enum { kStatic = 0, kBEuler = 1, kWarp = 2, kNewmark = 3 };

struct TetParam {
  double lam, myu;            // of unit modulus (kStatic) or the material's
  double rho, g[3], dt, beta;
  const double *young;        // kStatic: per tet
  const double *rot, *acc;    // kWarp, kNewmark
  const double *disp, *velo;  // dynamic modes; kStatic: disp or null
};

__device__ __forceinline__ void tet_grad(const double *__restrict__ geo, unsigned e, unsigned a, double d[3],
                                         double *vol) {
  const double2 *g = reinterpret_cast<const double2 *>(geo + (size_t)e * 16);
  const double2 xy = __ldg(g + 2 * a), zv = __ldg(g + 2 * a + 1);
  d[0] = xy.x;
  d[1] = xy.y;
  d[2] = zv.x;
  *vol = a == 0 ? zv.y : __ldg(geo + (size_t)e * 16 + 3);
}

// K_ij of the summed X (see above).
__device__ __forceinline__ void tet_block(const double X[9], double lam, double myu, double k[9]) {
  const double d = myu * (X[0] + X[4] + X[8]);
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) k[r * 3 + c] = lam * X[r * 3 + c] + myu * X[c * 3 + r] + (r == c ? d : 0.0);
}

__device__ __forceinline__ void rotate_block(const double R[9], double k[9]) {  // k <- R k R^T
  double t[9];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) t[r * 3 + c] = k[r * 3] * R[c * 3] + k[r * 3 + 1] * R[c * 3 + 1] + k[r * 3 + 2] * R[c * 3 + 2];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) k[r * 3 + c] = R[r * 3] * t[c] + R[r * 3 + 1] * t[3 + c] + R[r * 3 + 2] * t[6 + c];
}

// One thread per edge: the blocks (i, j) and (j, i).
template <int MODE>
__global__ void __launch_bounds__(128) k_tet_edges(unsigned nedge, const unsigned *__restrict__ eslot,
                                                   const unsigned *__restrict__ eoff, unsigned total,
                                                   const unsigned *__restrict__ elist,
                                                   const unsigned *__restrict__ slot,
                                                   const unsigned *__restrict__ tet, const double *__restrict__ geo,
                                                   const TetParam p, double *vcrs) {
  const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nedge) return;
  const unsigned l0 = eoff[k], l1 = k + 1 < nedge ? eoff[k + 1] : total;
  double X[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, vsum = 0.0;
  unsigned code = 0;
  for (unsigned l = l0; l < l1; ++l) {
    code = elist[l];
    const unsigned e = code >> 4;
    double a[3], b[3], vol;
    tet_grad(geo, e, (code >> 2) & 3u, a, &vol);
    tet_grad(geo, e, code & 3u, b, &vol);
    const double w = MODE == kStatic ? p.young[e] * vol : vol;
    if (MODE == kNewmark) vsum += vol;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const double wa = w * a[r];
#pragma unroll
      for (int c = 0; c < 3; ++c) X[r * 3 + c] += wa * b[c];
    }
  }
  double kij[9], kji[9];
  tet_block(X, p.lam, p.myu, kij);
  if (MODE == kNewmark) {
    const double s = p.beta * p.dt * p.dt, m = p.rho * vsum * 0.05;
#pragma unroll
    for (int q = 0; q < 9; ++q) kij[q] = (q % 4 == 0 ? m : 0.0) + s * kij[q];
  }
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) kji[r * 3 + c] = kij[c * 3 + r];
  const unsigned e = code >> 4, a = (code >> 2) & 3u, b = code & 3u;
  if (MODE == kWarp) {
    double R[9];
    const double *Ri = p.rot + (size_t)tet[(size_t)e * 4 + a] * 9, *Rj = p.rot + (size_t)tet[(size_t)e * 4 + b] * 9;
#pragma unroll
    for (int q = 0; q < 9; ++q) R[q] = Ri[q];
    rotate_block(R, kij);
#pragma unroll
    for (int q = 0; q < 9; ++q) R[q] = Rj[q];
    rotate_block(R, kji);
  }
  double *up = vcrs + (size_t)eslot[k] * 9, *lo = vcrs + (size_t)slot[(size_t)e * 16 + b * 4 + a] * 9;
#pragma unroll
  for (int q = 0; q < 9; ++q) up[q] += kij[q];
#pragma unroll
  for (int q = 0; q < 9; ++q) lo[q] += kji[q];
}

// S = vol (lam tr(G) I + myu (G + G^T)), G = sum_b w_b dN_b^T: the nodal forces
// K_e w are S dN_a. Stored as {xx, yy, zz, xy, yz, zx}.
__device__ __forceinline__ void tet_stress(const double G[9], double lam, double myu, double S[6]) {
  const double t = lam * (G[0] + G[4] + G[8]);
  S[0] = t + 2.0 * myu * G[0];
  S[1] = t + 2.0 * myu * G[4];
  S[2] = t + 2.0 * myu * G[8];
  S[3] = myu * (G[1] + G[3]);
  S[4] = myu * (G[5] + G[7]);
  S[5] = myu * (G[6] + G[2]);
}

// One thread per tet: S of w = u (kStatic), u + dt v (kBEuler), u + dt v + dt^2/2 acc (kNewmark);
// kWarp: G of w = u + dt v itself, nine values, as each node of the tet turns it its own way.
template <int MODE>
__global__ void __launch_bounds__(128) k_tet_stress(size_t ntet, const unsigned *__restrict__ tet,
                                                    const double *__restrict__ geo, const TetParam p,
                                                    double *__restrict__ stress) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < ntet; e += (size_t)gridDim.x * blockDim.x) {
    double G[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, vol = 0.0;
#pragma unroll
    for (unsigned b = 0; b < 4; ++b) {
      const size_t n = (size_t)tet[e * 4 + b] * 3;
      double d[3], v;
      tet_grad(geo, (unsigned)e, b, d, &v);
      if (b == 0) vol = v;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        double w = p.disp[n + r];
        if (MODE != kStatic) w += p.dt * p.velo[n + r];
        if (MODE == kNewmark) w += 0.5 * p.dt * p.dt * p.acc[n + r];
#pragma unroll
        for (int c = 0; c < 3; ++c) G[r * 3 + c] += w * d[c];
      }
    }
    if (MODE == kWarp) {
#pragma unroll
      for (int q = 0; q < 9; ++q) stress[e * 9 + q] = G[q];
      continue;
    }
    const double w = MODE == kStatic ? p.young[e] * vol : vol;
    double S[6];
    tet_stress(G, w * p.lam, w * p.myu, S);
    double2 *o = reinterpret_cast<double2 *>(stress + e * 6);
    o[0] = make_double2(S[0], S[1]);
    o[1] = make_double2(S[2], S[3]);
    o[2] = make_double2(S[4], S[5]);
  }
}

// The diagonal block and the right-hand side of a node, summed by LN lanes
// (each takes every LN-th tet; a shuffle tree adds their sums). A thread per
// node of a small mesh leaves most of the machine idle while each runs some 24
// tets of FP64 one after the other: LN doubles until there is a warp for each
// SM quarter (an FP64 warp instruction takes a quarter 64 cycles, so more warps
// would not help).
template <int MODE, int LN>
__global__ void __launch_bounds__(128) k_tet_nodes(unsigned np, const unsigned *__restrict__ noff, unsigned total,
                                                   const unsigned *__restrict__ nlist,
                                                   const unsigned *__restrict__ tet, const double *__restrict__ geo,
                                                   const double *__restrict__ stress, const TetParam p, double *vdia,
                                                   double *rhs) {
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x, sub = t % LN, i0 = t / LN;
  const unsigned i = i0 < np ? i0 : np - 1;
  const unsigned l0 = noff[i], l1 = i + 1 < np ? noff[i + 1] : total;
  double X[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, vsum = 0.0, vmass = 0.0, f[3] = {0, 0, 0}, macc[3] = {0, 0, 0};
  double skew[3] = {0, 0, 0};
  double R[9];
  if (MODE == kWarp) {
#pragma unroll
    for (int q = 0; q < 9; ++q) R[q] = p.rot[(size_t)i * 9 + q];
  }
  for (unsigned l = l0 + sub; l < l1; l += LN) {
    const unsigned code = nlist[l], e = code >> 4, ia = (code >> 2) & 3u, ib = code & 3u;
    double a[3], vol;
    tet_grad(geo, e, ia, a, &vol);
    const double w = MODE == kStatic ? p.young[e] * vol : vol;
    double b[3] = {a[0], a[1], a[2]};
    // a tet that names the node twice: K_ab joins the diagonal (kStatic), or the
    // (a, a) block once more (the dynamic forms), as the reference's Merge does
    if (ia != ib && MODE == kStatic) tet_grad(geo, e, ib, b, &vol);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const double wa = w * a[r];
#pragma unroll
      for (int c = 0; c < 3; ++c)
        if (c >= r) X[r * 3 + c] += wa * b[c];
    }
    if (MODE == kStatic && ia != ib) {  // the lower part's excess over the upper one
      skew[0] += w * (a[1] * b[0] - a[0] * b[1]);
      skew[1] += w * (a[2] * b[0] - a[0] * b[2]);
      skew[2] += w * (a[2] * b[1] - a[1] * b[2]);
    }
    vmass += vol;
    if (ia != ib) continue;
    vsum += vol;
    if (MODE == kWarp) {
      // G = sum_q R^T (P_q + u_q + dt v_q - R P_q) dN_q^T = R^T (I + U - R), as
      // sum_q P_q dN_q^T = I, with U of k_tet_stress: 27 products instead of 130
      double H[9], G[9];
#pragma unroll
      for (int q = 0; q < 9; ++q) H[q] = __ldg(stress + (size_t)e * 9 + q) + ((q % 4 == 0 ? 1.0 : 0.0) - R[q]);
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) G[r * 3 + c] = R[r] * H[c] + R[3 + r] * H[3 + c] + R[6 + r] * H[6 + c];
      double S[6];
      tet_stress(G, vol * p.lam, vol * p.myu, S);
      f[0] += S[0] * a[0] + S[3] * a[1] + S[5] * a[2];
      f[1] += S[3] * a[0] + S[1] * a[1] + S[4] * a[2];
      f[2] += S[5] * a[0] + S[4] * a[1] + S[2] * a[2];
    } else if (stress) {
      const double2 *o = reinterpret_cast<const double2 *>(stress + (size_t)e * 6);
      const double2 s0 = __ldg(o), s1 = __ldg(o + 1), s2 = __ldg(o + 2);
      f[0] += s0.x * a[0] + s1.y * a[1] + s2.y * a[2];
      f[1] += s1.y * a[0] + s0.y * a[1] + s2.x * a[2];
      f[2] += s2.y * a[0] + s2.x * a[1] + s1.x * a[2];
    }
    if (MODE == kNewmark) {
#pragma unroll
      for (unsigned q = 0; q < 4; ++q) {
        const double *x = p.acc + (size_t)tet[(size_t)e * 4 + q] * 3;
        const double m = q == ia ? 2.0 * vol : vol;
#pragma unroll
        for (int r = 0; r < 3; ++r) macc[r] += m * x[r];
      }
    }
  }
  if (LN > 1) {
    auto add = [](double &v) {
#pragma unroll
      for (int o = 1; o < LN; o *= 2) v += __shfl_xor_sync(0xffffffffu, v, o);
    };
#pragma unroll
    for (int q = 0; q < 9; ++q)
      if (q % 3 >= q / 3) add(X[q]);
    add(vmass), add(vsum);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      add(f[r]);
      if (MODE == kStatic) add(skew[r]);
      if (MODE == kNewmark) add(macc[r]);
    }
  }
  if (sub != 0 || i0 >= np || l0 == l1) return;
  X[3] = X[1] + skew[0];
  X[6] = X[2] + skew[1];
  X[7] = X[5] + skew[2];
  double k[9];
  tet_block(X, p.lam, p.myu, k);
  if (MODE == kWarp) rotate_block(R, k);
  double m = 0.0;
  if (MODE == kBEuler || MODE == kWarp) m = p.rho * vmass * 0.25 / (p.dt * p.dt);
  if (MODE == kNewmark) {
    const double s = p.beta * p.dt * p.dt;
#pragma unroll
    for (int q = 0; q < 9; ++q) k[q] *= s;
    m = p.rho * vmass * 0.1;
  }
  double *dst = vdia + (size_t)i * 9;
#pragma unroll
  for (int q = 0; q < 9; ++q) dst[q] += k[q] + (q % 4 == 0 ? m : 0.0);
  if (MODE == kWarp) {
    const double t0 = f[0], t1 = f[1], t2 = f[2];
#pragma unroll
    for (int r = 0; r < 3; ++r) f[r] = R[r * 3] * t0 + R[r * 3 + 1] * t1 + R[r * 3 + 2] * t2;
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    double q = vsum * p.rho * p.g[r] * 0.25 - f[r];
    if (MODE == kNewmark) q -= p.rho * 0.05 * macc[r];
    if (MODE == kBEuler || MODE == kWarp) q /= p.dt;
    rhs[(size_t)i * 3 + r] += q;
  }
}

// The scalar matrix of EMat_Poisson_Tet3D (include/delfem2/fem_poisson.cpp:
// 163-194), K_e[a][b] = alpha vol (dN_a . dN_b): one thread per edge, and per
// node (b_i += source vol/4 - sum_b K_ab val_b; a pair of a tet that names a
// node twice adds the (a, a) entry again, as the reference's Merge does).
__global__ void __launch_bounds__(128) k_poisson_edges(unsigned nedge, const unsigned *__restrict__ eslot,
                                                       const unsigned *__restrict__ eoff, unsigned total,
                                                       const unsigned *__restrict__ elist,
                                                       const unsigned *__restrict__ slot,
                                                       const double *__restrict__ geo, double alpha, double *vcrs) {
  const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nedge) return;
  const unsigned l0 = eoff[k], l1 = k + 1 < nedge ? eoff[k + 1] : total;
  double x = 0.0;
  unsigned code = 0;
  for (unsigned l = l0; l < l1; ++l) {
    code = elist[l];
    double a[3], b[3], vol;
    tet_grad(geo, code >> 4, (code >> 2) & 3u, a, &vol);
    tet_grad(geo, code >> 4, code & 3u, b, &vol);
    x += vol * (a[0] * b[0] + a[1] * b[1] + a[2] * b[2]);
  }
  x *= alpha;
  vcrs[eslot[k]] += x;
  vcrs[slot[(size_t)(code >> 4) * 16 + (code & 3u) * 4 + ((code >> 2) & 3u)]] += x;
}

__global__ void __launch_bounds__(128) k_poisson_nodes(unsigned np, const unsigned *__restrict__ noff, unsigned total,
                                                       const unsigned *__restrict__ nlist,
                                                       const unsigned *__restrict__ tet,
                                                       const double *__restrict__ geo, double alpha, double source,
                                                       const double *__restrict__ val, double *vdia, double *rhs) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const unsigned l0 = noff[i], l1 = i + 1 < np ? noff[i + 1] : total;
  if (l0 == l1) return;
  double x = 0.0, res = 0.0, vsum = 0.0;
  for (unsigned l = l0; l < l1; ++l) {
    const unsigned code = nlist[l], e = code >> 4, ia = (code >> 2) & 3u;
    double a[3], vol;
    tet_grad(geo, e, ia, a, &vol);
    x += vol * (a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
    if (ia != (code & 3u)) continue;
    vsum += vol;
    if (val) {
      double g[3] = {0, 0, 0};
#pragma unroll
      for (unsigned q = 0; q < 4; ++q) {
        const double u = val[tet[(size_t)e * 4 + q]];
        double d[3], v;
        tet_grad(geo, e, q, d, &v);
#pragma unroll
        for (int r = 0; r < 3; ++r) g[r] += u * d[r];
      }
      res += vol * (a[0] * g[0] + a[1] * g[1] + a[2] * g[2]);
    }
  }
  vdia[i] += alpha * x;
  rhs[i] += source * vsum * 0.25 - alpha * res;
}

// dL/dE_e = -lam_e^T (K_e / E_e) u_e with G(v)[r][c] = sum_k v_k[r] dN_k[c]:
// lam^T K_e u = vol (lambda1 tr(GL) tr(GU) + myu1 (tr(GL GU) + GL:GU)),
// lambda1 = nu/((1+nu)(1-2nu)), myu1 = 1/(2(1+nu)) (the moduli at E = 1).
__global__ void k_tet_dLdE(size_t ntet, const unsigned *__restrict__ tet, const double *__restrict__ geo, double nu,
                           const double *__restrict__ u, const double *__restrict__ lamv, double *__restrict__ out) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < ntet; e += (size_t)gridDim.x * blockDim.x) {
    unsigned nd[4];
    double dN[4][3], vol = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      double v;
      nd[k] = tet[e * 4 + k];
      tet_grad(geo, (unsigned)e, k, dN[k], &v);
      if (k == 0) vol = v;
    }
    double GL[3][3] = {{0}}, GU[3][3] = {{0}};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double *lk = lamv + (size_t)nd[k] * 3, *uk = u + (size_t)nd[k] * 3;
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          GL[r][c] += lk[r] * dN[k][c];
          GU[r][c] += uk[r] * dN[k][c];
        }
    }
    const double lam1 = nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
    const double myu1 = 1.0 / (2.0 * (1.0 + nu));
    double tr_prod = 0.0, frob = 0.0;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        tr_prod += GL[r][c] * GU[c][r];
        frob += GL[r][c] * GU[r][c];
      }
    const double trL = GL[0][0] + GL[1][1] + GL[2][2], trU = GU[0][0] + GU[1][1] + GU[2][2];
    out[e] = -vol * (lam1 * trL * trU + myu1 * (tr_prod + frob));
  }
}

}  // namespace dfm2g

using namespace dfm2g;

static int scan_exclusive(const unsigned *a, unsigned n, int flag, unsigned *out, unsigned *sums, unsigned *total) {
  const unsigned tiles = (n + kScanTile - 1) / kScanTile;
  k_scan_tile<<<tiles, 256, 0, stream()>>>(a, n, flag, nullptr, nullptr, sums);
  k_scan_sums<<<1, 1024, 0, stream()>>>(sums, tiles, total);
  k_scan_tile<<<tiles, 256, 0, stream()>>>(a, n, flag, sums, out, nullptr);
  note_launches(3);
  DFM2G_LAUNCH_CHECK();
  return DFM2G_OK;
}

// The gather lists and the tets' geometry (see the top of the file).
static int tet_lists_build(dfm2g_tetmesh_s *t, const dfm2g_bsr_s *m) {
  const unsigned np = (unsigned)t->np, nnz = (unsigned)m->nnz;
  DFM2G_TRY(t->geo.resize(t->ntet * 16 + 2));
  // the stresses' workspace for every mode, so that no assembly allocates (it may
  // be captured) and none moves a buffer that a captured one still writes
  if (m->ndim == 3) DFM2G_TRY(t->stress.resize(t->ntet * 9 + 2));
  DFM2G_TRY(t->noff.resize(np + 1));
  if (t->ntet == 0) return DFM2G_OK;
  const unsigned grid = ctx().num_sms * 16;
  k_tet_geo<<<grid, 256, 0, stream()>>>(t->ntet, t->tet.p, t->xyz.p, t->geo.p);
  // scratch: counts, first entries and ranks of the slots, counts of the nodes, tile sums, three totals
  const size_t most = std::max((size_t)nnz, (size_t)np);
  DevBuf<unsigned> tmp;
  DFM2G_TRY(tmp.resize(3 * (size_t)nnz + np + most / kScanTile + 8));
  unsigned *count = tmp.p, *ncount = count + nnz, *at = ncount + np, *rank = at + nnz, *totals = rank + nnz,
           *sums = totals + 3;
  DFM2G_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned) * ((size_t)nnz + np), stream()));
  DFM2G_CUDA(cudaMemsetAsync(totals, 0, sizeof(unsigned) * 3, stream()));
  k_tet_lists<<<grid, 256, 0, stream()>>>(t->ntet, t->tet.p, t->slot.p, 0, count, ncount, nullptr, nullptr);
  DFM2G_TRY(scan_exclusive(ncount, np, 0, t->noff.p, sums, totals));
  if (nnz) {
    DFM2G_TRY(scan_exclusive(count, nnz, 1, rank, sums, totals + 1));
    DFM2G_TRY(scan_exclusive(count, nnz, 0, at, sums, totals + 2));
  }
  unsigned h[3];
  DFM2G_CUDA(cudaMemcpyAsync(h, totals, sizeof(h), cudaMemcpyDeviceToHost, stream()));
  DFM2G_CUDA(cudaStreamSynchronize(stream()));
  t->nnode_entries = h[0];
  t->nedge = h[1];
  t->nedge_entries = h[2];
  DFM2G_TRY(t->nlist.resize((size_t)h[0] + 1));
  DFM2G_TRY(t->elist.resize((size_t)h[2] + 1));
  DFM2G_TRY(t->eslot.resize((size_t)h[1] + 1));
  DFM2G_TRY(t->eoff.resize((size_t)h[1] + 1));
  if (nnz) k_tet_edges_compact<<<grid, 256, 0, stream()>>>(nnz, count, at, rank, t->eslot.p, t->eoff.p);
  // the fill advances the slots' first entries and a copy of the nodes'
  DFM2G_CUDA(cudaMemcpyAsync(ncount, t->noff.p, sizeof(unsigned) * np, cudaMemcpyDeviceToDevice, stream()));
  k_tet_lists<<<grid, 256, 0, stream()>>>(t->ntet, t->tet.p, t->slot.p, 1, at, ncount, t->elist.p, t->nlist.p);
  k_sort_lists<<<grid, 128, 0, stream()>>>(np, t->noff.p, t->nnode_entries, t->nlist.p);
  if (t->nedge) k_sort_lists<<<grid, 128, 0, stream()>>>(t->nedge, t->eoff.p, t->nedge_entries, t->elist.p);
  note_launches(6);
  DFM2G_LAUNCH_CHECK();
  DFM2G_CUDA(cudaStreamSynchronize(stream()));
  return DFM2G_OK;
}

template <int MODE>
static int tet_assemble(dfm2g_tetmesh_s *t, dfm2g_bsr_s *m, const TetParam &p, double *b) {
  if (t->ntet == 0) return DFM2G_OK;
  const double *stress = nullptr;
  if (p.disp) {
    k_tet_stress<MODE><<<blocks_for(t->ntet, 128), 128, 0, stream()>>>(t->ntet, t->tet.p, t->geo.p, p, t->stress.p);
    stress = t->stress.p;
  }
  if (t->nedge)
    k_tet_edges<MODE><<<blocks_for(t->nedge, 128), 128, 0, stream()>>>(t->nedge, t->eslot.p, t->eoff.p,
                                                                      t->nedge_entries, t->elist.p, t->slot.p,
                                                                      t->tet.p, t->geo.p, p, m->vcrs.p);
  const size_t quarters = (size_t)ctx().num_sms * 4 * 32;  // threads at a warp for each SM quarter
  auto nodes = [&](auto *kernel, unsigned lanes) {
    kernel<<<blocks_for(t->np * lanes, 128), 128, 0, stream()>>>((unsigned)t->np, t->noff.p, t->nnode_entries,
                                                                t->nlist.p, t->tet.p, t->geo.p, stress, p, m->vdia.p,
                                                                b);
  };
  if (t->np * 8 <= quarters)
    nodes(k_tet_nodes<MODE, 8>, 8);
  else if (t->np * 4 <= quarters)
    nodes(k_tet_nodes<MODE, 4>, 4);
  else if (t->np * 2 <= quarters)
    nodes(k_tet_nodes<MODE, 2>, 2);
  else
    nodes(k_tet_nodes<MODE, 1>, 1);
  note_launches(stress ? 3 : 2);
  DFM2G_LAUNCH_CHECK();
  m->f32_valid = false;
  return DFM2G_OK;
}

extern "C" {

int dfm2g_tetmesh_create(dfm2g_tetmesh *out, dfm2g_bsr m, const double *xyz, size_t np, const unsigned *tet,
                         size_t ntet) try {
  if (!out) return fail(DFM2G_ERR_ARG, "tetmesh_create: null out");
  if (!m || !m->has_pattern) return fail(DFM2G_ERR_STATE, "tetmesh_create: matrix has no pattern");
  if (m->ndim == 2) return fail(DFM2G_ERR_UNSUPPORTED, "tetmesh_create: 2x2 blocks (tets take 1x1 or 3x3)");
  if (np != m->nblk) return fail(DFM2G_ERR_ARG, "tetmesh_create: np (%zu) != matrix blocks (%u)", np, m->nblk);
  if ((ntet && !tet) || (np && !xyz)) return fail(DFM2G_ERR_ARG, "tetmesh_create: null mesh array");
  if (ntet > 0xFFFFFFFFull / 16) return fail(DFM2G_ERR_ARG, "tetmesh_create: too many tets");
  DFM2G_TRY(ensure_context());
  auto *t = new dfm2g_tetmesh_s();
  t->np = np;
  t->ntet = ntet;
  t->nblk = m->nblk;
  t->bsr = m;
  t->pattern_version = m->pattern_version;
  std::vector<unsigned> by_color;
  int s = color_elements(tet, ntet, 4, np, by_color, t->color_start);
  if (s == DFM2G_OK) s = t->xyz.resize(np * 3 + 1);
  if (s == DFM2G_OK) s = t->tet.resize(ntet * 4 + 1);
  if (s == DFM2G_OK) s = t->slot.resize(ntet * 16 + 1);
  if (s == DFM2G_OK && np &&
      cudaMemcpyAsync(t->xyz.p, xyz, sizeof(double) * np * 3, cudaMemcpyHostToDevice, stream()) != cudaSuccess)
    s = fail(DFM2G_ERR_CUDA, "tetmesh_create: copy xyz");
  if (s == DFM2G_OK && ntet &&
      cudaMemcpyAsync(t->tet.p, tet, sizeof(unsigned) * ntet * 4, cudaMemcpyHostToDevice, stream()) != cudaSuccess)
    s = fail(DFM2G_ERR_CUDA, "tetmesh_create: copy tets");
  if (s == DFM2G_OK) s = build_slot_map(t->tet.p, ntet, 4, m, t->slot.p);
  if (s == DFM2G_OK) s = tet_lists_build(t, m);
  if (s != DFM2G_OK) {
    delete t;
    return s;
  }
  *out = t;
  return DFM2G_OK;
} catch (...) {
  return host_failure();
}

int dfm2g_tetmesh_destroy(dfm2g_tetmesh t) try {
  if (t) {
    cudaStreamSynchronize(stream());
    delete t;
  }
  return DFM2G_OK;
} catch (...) {
  return host_failure();
}

int dfm2g_tetmesh_info(dfm2g_tetmesh t, unsigned *ncolor, size_t *ntet) try {
  if (!t) return fail(DFM2G_ERR_ARG, "null tetmesh");
  if (ncolor) *ncolor = t->color_start.empty() ? 0 : (unsigned)t->color_start.size() - 1;
  if (ntet) *ntet = t->ntet;
  return DFM2G_OK;
} catch (...) {
  return host_failure();
}

int dfm2g_tetmesh_assemble_linear(dfm2g_tetmesh t, dfm2g_bsr m, const double *young, double nu, double rho,
                                  const double *g, const double *disp, double *b, int mem) try {
  if (!t || !m) return fail(DFM2G_ERR_ARG, "assemble: null handle");
  if (m != t->bsr || m->pattern_version != t->pattern_version)
    return fail(DFM2G_ERR_STATE, "assemble: matrix pattern differs from the one the mesh was mapped to");
  DFM2G_TRY(require_3x3(m, "tetmesh_assemble_linear"));
  if (!young || !g || !b) return fail(DFM2G_ERR_ARG, "assemble: null argument");
  VecArg<double> ay, ad, ab;
  DFM2G_TRY(ay.in(young, t->ntet, mem, true));
  if (disp) DFM2G_TRY(ad.in(disp, t->np * 3, mem, true));
  DFM2G_TRY(ab.in(b, t->np * 3, mem, true));
  TetParam p{};
  p.lam = nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
  p.myu = 1.0 / (2.0 * (1.0 + nu));
  p.rho = rho;
  for (int d = 0; d < 3; ++d) p.g[d] = g[d];
  p.young = ay.dev();
  p.disp = disp ? ad.dev() : nullptr;
  DFM2G_TRY(tet_assemble<kStatic>(t, m, p, ab.dev()));
  return ab.copy_back();
} catch (...) {
  return host_failure();
}

int dfm2g_tetmesh_assemble_poisson(dfm2g_tetmesh t, dfm2g_bsr m, double alpha, double source, const double *val,
                                   double *b, int mem) try {
  if (!t || !m) return fail(DFM2G_ERR_ARG, "assemble_poisson: null handle");
  if (m != t->bsr || m->pattern_version != t->pattern_version)
    return fail(DFM2G_ERR_STATE, "assemble_poisson: matrix pattern differs from the one the mesh was mapped to");
  if (m->ndim != 1) return fail(DFM2G_ERR_UNSUPPORTED, "assemble_poisson: needs a scalar (ndim 1) matrix");
  if (!b) return fail(DFM2G_ERR_ARG, "assemble_poisson: null b");
  VecArg<double> av, ab;
  if (val) DFM2G_TRY(av.in(val, t->np, mem, true));
  DFM2G_TRY(ab.in(b, t->np, mem, true));
  if (t->ntet) {
    if (t->nedge)
      k_poisson_edges<<<blocks_for(t->nedge, 128), 128, 0, stream()>>>(t->nedge, t->eslot.p, t->eoff.p,
                                                                      t->nedge_entries, t->elist.p, t->slot.p,
                                                                      t->geo.p, alpha, m->vcrs.p);
    k_poisson_nodes<<<blocks_for(t->np, 128), 128, 0, stream()>>>((unsigned)t->np, t->noff.p, t->nnode_entries,
                                                                 t->nlist.p, t->tet.p, t->geo.p, alpha, source,
                                                                 val ? av.dev() : nullptr, m->vdia.p, ab.dev());
    note_launches(2);
    DFM2G_LAUNCH_CHECK();
  }
  m->f32_valid = false;
  return ab.copy_back();
} catch (...) {
  return host_failure();
}

static int tet_dynamic(dfm2g_tetmesh t, dfm2g_bsr m, int mode, double myu, double lambda, double rho,
                       const double *g, double dt, double beta, const double *disp, const double *velo,
                       const double *third, double *b, int mem, const char *what) {
  if (!t || !m) return fail(DFM2G_ERR_ARG, "%s: null handle", what);
  if (m != t->bsr || m->pattern_version != t->pattern_version)
    return fail(DFM2G_ERR_STATE, "%s: matrix pattern differs from the one the mesh was mapped to", what);
  DFM2G_TRY(require_3x3(m, what));
  if (!g || !b || !disp || !velo || (mode != kBEuler && !third)) return fail(DFM2G_ERR_ARG, "%s: null argument", what);
  if (!(dt > 0)) return fail(DFM2G_ERR_ARG, "%s: dt must be positive", what);
  VecArg<double> ad, av, a3, ab;
  DFM2G_TRY(ad.in(disp, t->np * 3, mem, true));
  DFM2G_TRY(av.in(velo, t->np * 3, mem, true));
  if (mode != kBEuler) DFM2G_TRY(a3.in(third, t->np * (mode == kWarp ? 9 : 3), mem, true));
  DFM2G_TRY(ab.in(b, t->np * 3, mem, true));
  TetParam p{};
  p.lam = lambda;
  p.myu = myu;
  p.rho = rho;
  for (int d = 0; d < 3; ++d) p.g[d] = g[d];
  p.dt = dt;
  p.beta = beta;
  p.disp = ad.dev();
  p.velo = av.dev();
  if (mode == kWarp) p.rot = a3.dev();
  if (mode == kNewmark) p.acc = a3.dev();
  if (mode == kBEuler)
    DFM2G_TRY(tet_assemble<kBEuler>(t, m, p, ab.dev()));
  else if (mode == kWarp)
    DFM2G_TRY(tet_assemble<kWarp>(t, m, p, ab.dev()));
  else
    DFM2G_TRY(tet_assemble<kNewmark>(t, m, p, ab.dev()));
  return ab.copy_back();
}

int dfm2g_tetmesh_assemble_beuler(dfm2g_tetmesh t, dfm2g_bsr m, double myu, double lambda, double rho,
                                  const double *g, double dt, const double *disp, const double *velo,
                                  const double *rot, double *b, int mem) try {
  return tet_dynamic(t, m, rot ? kWarp : kBEuler, myu, lambda, rho, g, dt, 0.0, disp, velo, rot, b, mem,
                     "tetmesh_assemble_beuler");
} catch (...) {
  return host_failure();
}

int dfm2g_tetmesh_assemble_newmark(dfm2g_tetmesh t, dfm2g_bsr m, double myu, double lambda, double rho,
                                   const double *g, double dt, double gamma, double beta, const double *disp,
                                   const double *velo, const double *acc, double *b, int mem) try {
  (void)gamma;  // unused by the reference's first-iteration element matrix as well
  return tet_dynamic(t, m, kNewmark, myu, lambda, rho, g, dt, beta, disp, velo, acc, b, mem,
                     "tetmesh_assemble_newmark");
} catch (...) {
  return host_failure();
}

int dfm2g_tetmesh_dLdE(dfm2g_tetmesh t, const double *young, double nu, const double *u, const double *lam,
                       double *dLdE, int mem) try {
  if (!t) return fail(DFM2G_ERR_ARG, "dLdE: null handle");
  (void)young;
  if (!u || !lam || !dLdE) return fail(DFM2G_ERR_ARG, "dLdE: null argument");
  VecArg<double> au, al, ao;
  DFM2G_TRY(au.in(u, t->np * 3, mem, true));
  DFM2G_TRY(al.in(lam, t->np * 3, mem, true));
  DFM2G_TRY(ao.in(dLdE, t->ntet, mem, false));
  if (t->ntet)
    k_tet_dLdE<<<blocks_for(t->ntet, 128, ctx().num_sms * 32), 128, 0, stream()>>>(t->ntet, t->tet.p, t->geo.p, nu,
                                                                                  au.dev(), al.dev(), ao.dev());
  DFM2G_LAUNCH_CHECK();
  return ao.copy_back();
} catch (...) {
  return host_failure();
}

}  // extern "C"
