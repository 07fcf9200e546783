// Whole smoothing passes of the smallest multigrid levels, one launch each.
//
// A smoother step on a level of a few thousand nodes is 0.3 us of work behind
// 2.3 us of launch, wait and first load (stencil.cu), and a V-cycle takes seven
// of them per level.  Here one CTA takes one column of cells (two node columns)
// and all radii, computes what its three steps need of the neighbouring columns
// itself -- 9, 5 and 2 columns, since a row reaches two columns to either side
// -- and so needs no other CTA between the steps: the pre-smoothing with its
// residual is one launch, the prolongation with the post-smoothing another.
// The lanes of a row keep its blocks in registers for all three applies,
// fetched before the wait; d goes through shared memory.  Sums are taken in the
// order of the single steps.
//
// The columns are computed 2.7 times over in the mean, which costs nothing as
// long as the level leaves the chip idle otherwise: one CTA per SM and at most
// one wave (halo_fits).  An inner iteration, with the single steps -> like this:
// 68 -> 60 us at 16x128 in FP64, 94 -> 82 at 32x256 and 262 -> 251 at 128x1024
// on the FP32 hierarchy.
#pragma once
#include "kernels.cuh"

namespace dp {

constexpr int kHaloDegree = 3;               // smoother steps that the columns below are made for
constexpr int kHaloCols = 13;                // node columns [-6, 6] around the core columns 0 and 1
// threads of a CTA: FP32 rows need 20 registers for their blocks, FP64 rows 40
template <typename T>
constexpr int halo_max_threads() { return sizeof(T) == 4 ? 1024 : 800; }
constexpr int kHaloMaxA = 41;                // largest A = 2 ncr + 1 with halo_warps(ncr) <= 32

// columns of rows around a CTA's cell: -4, -2, 0, 2, 4 for the even classes, -3, -1, 1, 3 for the odd ones
__host__ __device__ constexpr int halo_rows(int c, int ncr) { return ((c & 1) ? ncr : ncr + 1) * (c < 2 ? 5 : 4); }
__host__ __device__ constexpr int halo_class_warps(int c, int ncr) {
  return (halo_rows(c, ncr) * st_lanes(c) + 31) / 32;
}
__host__ __device__ constexpr int halo_warps(int ncr) {
  return halo_class_warps(0, ncr) + halo_class_warps(1, ncr) + halo_class_warps(2, ncr) + halo_class_warps(3, ncr);
}
static_assert(halo_warps((kHaloMaxA - 1) / 2) == 32 && halo_warps((kHaloMaxA + 1) / 2) > 32, "largest halo level");

// The level fits one wave of column CTAs.  From three columns of cells on, the
// 13 node columns wrap at most once.
template <typename T>
static bool halo_fits(const Level& g) {
  const int threads = 32 * halo_warps(g.ncr);
  if (threads > halo_max_threads<T>() || g.nct < 4) return false;
  return (int64_t)g.nct <= 148 * (int64_t)(halo_max_threads<T>() / threads);
}

// One row's share of a lane: 5 blocks, where their vectors lie in the 13-column
// patch, and the row itself.
template <typename T>
struct HaloRow {
  Blk2<T> k[5];
  int nb[5];        // patch index of each neighbour (the row itself where the block is zero)
  int node, own;    // node of the level, patch index
  int off, npw;     // column relative to the CTA's first; rows per warp
  bool store;       // this lane holds the row's result

  template <int C>
  __device__ __forceinline__ void init(const T* S, int w, int ncr, int nct) {
    constexpr int NE = st_entries(C), LN = st_lanes(C), PER = 5, NPW = 32 / LN, PA = C & 1, PB = C >> 1;
    const int lane = threadIdx.x & 31, sub = lane / NPW, i0 = w * NPW + lane % NPW;
    const int cnt = halo_rows(C, ncr), nA = PA ? ncr : ncr + 1, A = 2 * ncr + 1;
    const int i = min(i0, cnt - 1);          // idle lanes repeat the last row
    const int col = i / nA, ia = i - col * nA;
    off = 2 * col - 4 + PB;
    int jb = (int)blockIdx.x + ((off - PB) >> 1);
    if (jb < 0) jb += nct;
    if (jb >= nct) jb -= nct;
    const int a = 2 * ia + PA;
    node = a + A * (2 * jb + PB);
    own = a + A * (off + 6);
    npw = NPW;
    store = i0 < cnt && sub == 0;
    const int64_t base = st_base(C, ncr, nct);
    const int n = st_nodes(C, ncr, nct);
#pragma unroll
    for (int q = 0; q < PER; ++q) k[q] = ld_block(S, base, min(sub * PER + q, NE - 1), n, jb * nA + ia);
    int da[PER], db[PER];
    bool ok[PER];
    ok[0] = lane_entry<C, 0>(sub, da[0], db[0]);
    ok[1] = lane_entry<C, 1>(sub, da[1], db[1]);
    ok[2] = lane_entry<C, 2>(sub, da[2], db[2]);
    ok[3] = lane_entry<C, 3>(sub, da[3], db[3]);
    ok[4] = lane_entry<C, 4>(sub, da[4], db[4]);
#pragma unroll
    for (int q = 0; q < PER; ++q)
      nb[q] = ok[q] && a + da[q] >= 0 && a + da[q] < A ? own + da[q] + A * db[q] : -1;
  }
  __device__ __forceinline__ void init(const T* S, int ncr, int nct) {
    const int w = threadIdx.x >> 5, w1 = halo_class_warps(0, ncr), w2 = w1 + halo_class_warps(1, ncr),
              w3 = w2 + halo_class_warps(2, ncr);
    if (w < w1) init<0>(S, w, ncr, nct);
    else if (w < w2) init<1>(S, w - w1, ncr, nct);
    else if (w < w3) init<2>(S, w - w2, ncr, nct);
    else init<3>(S, w - w3, ncr, nct);
  }
  // r -= (A v)(row), v in the patch; every lane of the warp takes part
  template <typename X2>
  __device__ __forceinline__ void subtract(const X2* v, T& r0, T& r1) const {
    T s0 = (T)0, s1 = (T)0;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      if (nb[q] >= 0) {
        const X2 u = v[nb[q]];
        s0 += k[q].k00 * u.x + k[q].k01 * u.y;
        s1 += k[q].k10 * u.x + k[q].k11 * u.y;
      }
    }
    if (npw == 8) {
      s0 += __shfl_xor_sync(0xffffffffu, s0, 8);
      s1 += __shfl_xor_sync(0xffffffffu, s1, 8);
    }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 16);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 16);
    r0 -= s0;
    r1 -= s1;
  }
};

// Node of the level behind patch index t < 13 A (column t / A - 6 of this CTA).
struct HaloNode {
  int a, b, n;
  __device__ __forceinline__ HaloNode(int t, int A, int B) {
    const int c = t / A;
    a = t - c * A;
    b = 2 * (int)blockIdx.x + c - 6;
    if (b < 0) b += B;
    if (b >= B) b -= B;
    n = a + A * b;
  }
};

// Pre-smoothing from x = 0 and the true residual: d0 = (1/theta) D^-1 b,
// r = b - A d0, d1, r -= A d1, d2, r -= A d2;  x = d0 + d1 + d2.
template <typename T>
__global__ void __launch_bounds__(halo_max_threads<T>()) k_halo_down(const T* S, const T* b, T* r, T* x,
                                                                     const T* dinv, const double* coef, int ncr,
                                                                     int nct) {
  grid_dep_launch();
  typedef typename V2<T>::T X2;
  __shared__ X2 sm[2][kHaloCols * kHaloMaxA];
  const int A = 2 * ncr + 1, t = threadIdx.x;
  HaloRow<T> row;
  row.init(S, ncr, nct);
  const HaloNode nd(min(t, kHaloCols * A - 1), A, 2 * nct);
  const NodeInv<T> di(dinv, row.node), dn(dinv, nd.n);
  const T it = (T)ld_early(coef), c1 = (T)ld_early(coef + 2), c2 = (T)ld_early(coef + 3),
          e1 = (T)ld_early(coef + 4), e2 = (T)ld_early(coef + 5);
  grid_dep_sync();
  const X2* b2 = reinterpret_cast<const X2*>(b);
  const X2 bt = b2[nd.n];
  X2 rv = b2[row.node];
  if (t < kHaloCols * A) {
    T z0, z1;
    dn.apply(bt.x, bt.y, z0, z1);
    X2 d;
    d.x = it * z0;
    d.y = it * z1;
    sm[0][t] = d;
  }
  __syncthreads();
  X2 xv, d;
  T z0, z1;
  row.subtract(sm[0], rv.x, rv.y);
  xv = sm[0][row.own];
  di.apply(rv.x, rv.y, z0, z1);
  d.x = c1 * xv.x + c2 * z0;
  d.y = c1 * xv.y + c2 * z1;
  xv.x += d.x;
  xv.y += d.y;
  if (row.store) sm[1][row.own] = d;
  __syncthreads();
  const bool on2 = row.off >= -2 && row.off <= 2;
  if (__any_sync(0xffffffffu, on2)) {
    row.subtract(sm[1], rv.x, rv.y);
    di.apply(rv.x, rv.y, z0, z1);
    d.x = e1 * d.x + e2 * z0;
    d.y = e1 * d.y + e2 * z1;
    xv.x += d.x;
    xv.y += d.y;
    if (row.store && on2) sm[0][row.own] = d;
  }
  __syncthreads();
  const bool on3 = row.off == 0 || row.off == 1;
  if (__any_sync(0xffffffffu, on3)) {
    row.subtract(sm[0], rv.x, rv.y);
    if (row.store && on3) {
      reinterpret_cast<X2*>(r)[row.node] = rv;
      reinterpret_cast<X2*>(x)[row.node] = xv;
    }
  }
}

// Prolongation and post-smoothing: x = xp + P xc, then three steps on A x = b.
// xp is another buffer than x, since the neighbours read it too.
template <typename T>
__global__ void __launch_bounds__(halo_max_threads<T>()) k_halo_up(const T* S, const T* b, const T* xc, const T* xp,
                                                                   T* x, const T* dinv, const double* coef, int ncr,
                                                                   int nct, int ncrc, int Ac, int Bc, int pin,
                                                                   RzOut rz) {
  grid_dep_launch();
  typedef typename V2<T>::T X2;
  __shared__ X2 sm[2][kHaloCols * kHaloMaxA];
  const int A = 2 * ncr + 1, t = threadIdx.x;
  HaloRow<T> row;
  row.init(S, ncr, nct);
  const NodeInv<T> di(dinv, row.node);
  const T it = (T)ld_early(coef), c1 = (T)ld_early(coef + 2), c2 = (T)ld_early(coef + 3),
          e1 = (T)ld_early(coef + 4), e2 = (T)ld_early(coef + 5);
  const HaloNode nd(min(t, kHaloCols * A - 1), A, 2 * nct);
  int cn[6];
  float w[6];   // dyadic fractions, exact in FP32
  {
    double wd[6];
    fine_node_weights(nd.a, nd.b, ncrc, Ac, Bc, cn, wd);
#pragma unroll
    for (int k = 0; k < 6; ++k) w[k] = (float)wd[k];
  }
  grid_dep_sync();
  X2 rv = reinterpret_cast<const X2*>(b)[row.node];
  if (t < kHaloCols * A) {
    X2 v = reinterpret_cast<const X2*>(xp)[nd.n];
    T s0 = (T)0, s1 = (T)0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const X2 u = reinterpret_cast<const X2*>(xc)[cn[k]];
      s0 += (T)w[k] * u.x;
      s1 += (T)w[k] * u.y;
    }
    if (!dof_fixed(nd.a, nd.b, 0, A - 1, pin)) v.x += s0;
    if (!dof_fixed(nd.a, nd.b, 1, A - 1, pin)) v.y += s1;
    sm[0][t] = v;
  }
  __syncthreads();
  X2 xv, d;
  T z0, z1;
  row.subtract(sm[0], rv.x, rv.y);
  xv = sm[0][row.own];
  di.apply(rv.x, rv.y, z0, z1);
  d.x = it * z0;
  d.y = it * z1;
  xv.x += d.x;
  xv.y += d.y;
  if (row.store) sm[1][row.own] = d;
  __syncthreads();
  const bool on2 = row.off >= -2 && row.off <= 2;
  if (__any_sync(0xffffffffu, on2)) {
    row.subtract(sm[1], rv.x, rv.y);
    di.apply(rv.x, rv.y, z0, z1);
    d.x = c1 * d.x + c2 * z0;
    d.y = c1 * d.y + c2 * z1;
    xv.x += d.x;
    xv.y += d.y;
    if (row.store && on2) sm[0][row.own] = d;
  }
  __syncthreads();
  double share = 0.0;
  const bool on3 = row.off == 0 || row.off == 1;
  if (__any_sync(0xffffffffu, on3)) {
    row.subtract(sm[0], rv.x, rv.y);
    di.apply(rv.x, rv.y, z0, z1);
    xv.x += e1 * d.x + e2 * z0;
    xv.y += e1 * d.y + e2 * z1;
    if (row.store && on3) {
      reinterpret_cast<X2*>(x)[row.node] = xv;
      if (rz.out) {
        const double2 rr = reinterpret_cast<const double2*>(rz.r)[row.node];
        share = rr.x * (double)xv.x + rr.y * (double)xv.y;
      }
    }
  }
  if (rz.out) block_add(rz.yy ? sqrt(*rz.yy) * share : share, rz.out);
}

}  // namespace dp
