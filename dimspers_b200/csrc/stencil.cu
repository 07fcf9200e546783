// Assembled node stencils of the small multigrid levels and the smoother
// steps on them, one kernel per Chebyshev step.
//
// On the levels that live in L2 an element-by-element step is two launches (the
// apply, which scatter-adds K_e d_e with atomics, and the vector step), and
// each launch costs more than its work.  Here the level's operator is stored
// per lattice node instead: the 2x2 blocks that couple it to its neighbours,
// 19 for a vertex (parity class 0) and 9 for the midpoints (classes 1..3), so
// a node's row of A d is a gather, the smoother's update of r, d and x follows
// in the same thread, and a step is one launch without atomics.  Its result
// does not depend on scheduling, so the deterministic mode uses it as it is
// (but for ST_STEP_RZ, whose sum takes an atomic per block: not in that mode).
// The price is 184 bytes of matrix per FP32 node where the element form has
// 156, which is why large levels keep the element form (kStencilMaxNodes).
#pragma once
#include <utility>

#include "kernels.cuh"
#include "mg.cuh"
#include "reduce.cuh"

namespace dp {

constexpr int kStMax = 19;   // blocks of a vertex row

// Neighbour offsets (radial, angular) of each parity class (a & 1) + 2 (b & 1),
// in the order in which the elements around an interior node meet them.
struct StencilOffsets {
  int n[4] = {0, 0, 0, 0};
  int da[4][kStMax] = {}, db[4][kStMax] = {};
};
constexpr int stencil_find(const StencilOffsets& t, int c, int da, int db) {
  for (int j = 0; j < t.n[c]; ++j)
    if (t.da[c][j] == da && t.db[c][j] == db) return j;
  return -1;
}
constexpr StencilOffsets make_stencil_offsets() {
  StencilOffsets t;
  for (int c = 0; c < 4; ++c)
    for (int ty = 0; ty < 2; ++ty)
      for (int k = 0; k < 6; ++k) {
        if ((loc_a(ty, k) & 1) != (c & 1) || (loc_b(ty, k) & 1) != (c >> 1)) continue;
        for (int m = 0; m < 6; ++m) {
          const int da = loc_a(ty, m) - loc_a(ty, k), db = loc_b(ty, m) - loc_b(ty, k);
          if (stencil_find(t, c, da, db) < 0) {
            t.da[c][t.n[c]] = da;
            t.db[c][t.n[c]] = db;
            ++t.n[c];
          }
        }
      }
  return t;
}
constexpr StencilOffsets kStencil = make_stencil_offsets();
static_assert(kStencil.n[0] == 19 && kStencil.n[1] == 9 && kStencil.n[2] == 9 && kStencil.n[3] == 9,
              "unexpected node coupling");

template <int C, int J>
struct StencilEntry {
  static constexpr int da = kStencil.da[C][J], db = kStencil.db[C][J];
};

__host__ __device__ constexpr int st_entries(int c) { return c == 0 ? 19 : 9; }
// lanes per node: at most 5 blocks per lane in every class
__host__ __device__ constexpr int st_lanes(int c) { return c == 0 ? 4 : 2; }
// nodes of a class, and its first node-block in the store (blocks of 4 T)
__host__ __device__ inline int st_nodes(int c, int ncr, int nct) { return ((c & 1) ? ncr : ncr + 1) * nct; }
__host__ __device__ inline int64_t st_base(int c, int ncr, int nct) {
  int64_t o = 0;
  for (int k = 0; k < c; ++k) o += (int64_t)st_entries(k) * st_nodes(k, ncr, nct);
  return o;
}
template <typename T>
inline size_t stencil_store(int ncr, int nct) { return (size_t)4 * st_base(4, ncr, nct); }

// One 2x2 block (k00, k01, k10, k11) of entry j of the i-th node of a class:
// FP32 one float4 per node, FP64 two double2 planes, nodes consecutive.
template <typename T>
struct Blk2 {
  T k00, k01, k10, k11;
};
__device__ __forceinline__ Blk2<float> ld_block(const float* S, int64_t base, int j, int n, int i) {
  const float4 v = ld_stream(reinterpret_cast<const float4*>(S) + base + (int64_t)j * n + i);
  return {v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ Blk2<double> ld_block(const double* S, int64_t base, int j, int n, int i) {
  const double2* p = reinterpret_cast<const double2*>(S) + 2 * (base + (int64_t)j * n) + i;
  const double2 u = ld_stream(p), v = ld_stream(p + n);
  return {u.x, u.y, v.x, v.y};
}
__device__ __forceinline__ void st_block(float* S, int64_t base, int j, int n, int i, const double* k) {
  reinterpret_cast<float4*>(S)[base + (int64_t)j * n + i] =
      make_float4((float)k[0], (float)k[1], (float)k[2], (float)k[3]);
}
__device__ __forceinline__ void st_block(double* S, int64_t base, int j, int n, int i, const double* k) {
  double2* p = reinterpret_cast<double2*>(S) + 2 * (base + (int64_t)j * n) + i;
  p[0] = make_double2(k[0], k[1]);
  p[n] = make_double2(k[2], k[3]);
}

// ---- assembly of the stencils from the packed element matrices ----------------------
// One thread per (node of class C): the elements around the node in a fixed
// order, sums in FP64, one rounding to T.  Blocks that would leave the annulus
// stay zero.
template <int C, int J, typename T>
__device__ __forceinline__ void stencil_sum(const T* __restrict__ K, int ia, int jb, int ncr, int nct, double acc[4]) {
  constexpr int PA = C & 1, PB = C >> 1, DA = StencilEntry<C, J>::da, DB = StencilEntry<C, J>::db;
  acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
#pragma unroll
  for (int ty = 0; ty < 2; ++ty) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        // all resolved at compile time: local node k is of class C, local node m at this offset from it
        if ((loc_a(ty, k) & 1) != PA || (loc_b(ty, k) & 1) != PB) continue;
        if (loc_a(ty, m) - loc_a(ty, k) != DA || loc_b(ty, m) - loc_b(ty, k) != DB) continue;
        const int ir = ia + ((PA - loc_a(ty, k)) >> 1);
        int it = jb + ((PB - loc_b(ty, k)) >> 1);
        if (ir < 0 || ir >= ncr) continue;
        if (it < 0) it += nct;
        const int64_t e = 2 * ((int64_t)ir + (int64_t)ncr * it) + ty;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int R = 2 * k + (q >> 1), Cc = 2 * m + (q & 1);
          acc[q] += (double)K[kidx<T>(R >= Cc ? packed_index12(R, Cc) : packed_index12(Cc, R), e)];
        }
      }
    }
  }
}

template <int C, int J, typename T>
__device__ __forceinline__ void stencil_entry(const T* __restrict__ K, T* S, int i, int ia, int jb, int ncr, int nct,
                                              int64_t base, int n) {
  double acc[4];
  stencil_sum<C, J, T>(K, ia, jb, ncr, nct, acc);
  st_block(S, base, J, n, i, acc);
}

template <int C, typename T, int... J>
__device__ __forceinline__ void stencil_row(const T* __restrict__ K, T* S, int i, int ncr, int nct,
                                            std::integer_sequence<int, J...>) {
  const int nA = (C & 1) ? ncr : ncr + 1;
  const int ia = i % nA, jb = i / nA;
  const int64_t base = st_base(C, ncr, nct);
  const int n = st_nodes(C, ncr, nct);
  (stencil_entry<C, J, T>(K, S, i, ia, jb, ncr, nct, base, n), ...);
}
template <int C, typename T>
__device__ __forceinline__ void stencil_node(const T* __restrict__ K, T* S, int i, int ncr, int nct) {
  stencil_row<C, T>(K, S, i, ncr, nct, std::make_integer_sequence<int, st_entries(C)>{});
}

template <typename T>
__global__ void __launch_bounds__(128) k_stencil_assemble(const T* __restrict__ K, T* S, int ncr, int nct) {
  const int c = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= st_nodes(c, ncr, nct)) return;
  if (c == 0) stencil_node<0, T>(K, S, i, ncr, nct);
  else if (c == 1) stencil_node<1, T>(K, S, i, ncr, nct);
  else if (c == 2) stencil_node<2, T>(K, S, i, ncr, nct);
  else stencil_node<3, T>(K, S, i, ncr, nct);
}

// ---- smoother steps -----------------------------------------------------------------
enum StepMode {
  ST_STEP = 0,      // r -= A v; d = c1 v + c2 D^-1 r; x += d           (v = the previous d)
  ST_STEP_X = 1,    // the same with x += v first (the step after ST_FIRST_X)
  ST_RESIDUAL = 2,  // r -= A v
  ST_STEP_RZ = 4,   // ST_STEP, then *rz.out += rz.r . s x
  ST_FIRST_X = 3,   // r = b - A v; d = (1/theta) D^-1 r                 (v = x, which gains d in the next step)
};

// D^-1 of a node, constant during a solve: fetched before the wait
template <typename T>
struct NodeInv {
  T a, b, c;
  __device__ __forceinline__ NodeInv(const T* __restrict__ dinv, int64_t n)
      : a(ld_early(dinv + 3 * n)), b(ld_early(dinv + 3 * n + 1)), c(ld_early(dinv + 3 * n + 2)) {}
  __device__ __forceinline__ void apply(T r0, T r1, T& z0, T& z1) const {
    z0 = a * r0 + b * r1;
    z1 = b * r0 + c * r1;
  }
};

// Adds the block's sum of v to *out (every thread of the block takes part).
__device__ __forceinline__ void block_add(double v, double* out) {
  __shared__ double part[32];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
    atomicAdd(out, t);
  }
}

// Offsets of entry sub * PER + Q of a class-C row, as selects between
// compile-time values (a table lookup by lane would serialise the warp).  Past
// the last entry: no offset, ok = false.
template <int C, int Q>
__device__ __forceinline__ bool lane_entry(int sub, int& da, int& db) {
  constexpr int NE = st_entries(C), PER = (NE + st_lanes(C) - 1) / st_lanes(C);
  constexpr int J0 = Q, J1 = PER + Q < NE ? PER + Q : 0, J2 = 2 * PER + Q < NE ? 2 * PER + Q : 0,
                J3 = 3 * PER + Q < NE ? 3 * PER + Q : 0;
  da = StencilEntry<C, J0>::da;
  db = StencilEntry<C, J0>::db;
  if (sub == 1) { da = StencilEntry<C, J1>::da; db = StencilEntry<C, J1>::db; }
  if (st_lanes(C) > 2) {
    if (sub == 2) { da = StencilEntry<C, J2>::da; db = StencilEntry<C, J2>::db; }
    if (sub == 3) { da = StencilEntry<C, J3>::da; db = StencilEntry<C, J3>::db; }
  }
  return sub * PER + Q < NE;
}

// returns the node's share of the sum of ST_STEP_RZ, without its scale
template <int C, int MODE, typename T>
__device__ __forceinline__ double smooth_node(const T* __restrict__ S, const T* v, const T* b, T* r, T* x, T* d,
                                            const T* __restrict__ dinv, const double* __restrict__ coef, int blk,
                                            int ncr, int nct, const double* rr) {
  typedef typename V2<T>::T X2;
  constexpr int NE = st_entries(C), LN = st_lanes(C), PER = (NE + LN - 1) / LN, NPW = 32 / LN;
  constexpr int PA = C & 1, PB = C >> 1;
  const int lane = threadIdx.x & 31, w = blk * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int sub = lane / NPW, i0 = w * NPW + lane % NPW;
  const int cnt = st_nodes(C, ncr, nct);
  const bool live = i0 < cnt;
  const int i = live ? i0 : cnt - 1;      // idle lanes repeat the last node (their result is not stored)
  const int nA = PA ? ncr : ncr + 1, A = 2 * ncr + 1, B = 2 * nct;
  const int jb = i / nA, a = 2 * (i - jb * nA) + PA, bb = 2 * jb + PB;
  const int n = a + A * bb, N = A * B;
  const int64_t base = st_base(C, ncr, nct);
  Blk2<T> k[PER];
  int nb[PER];
#pragma unroll
  for (int q = 0; q < PER; ++q) k[q] = ld_block(S, base, min(sub * PER + q, NE - 1), cnt, i);
  int da[PER], db[PER];
  bool ok[PER];
  static_assert(PER == 5, "five entries per lane");
  ok[0] = lane_entry<C, 0>(sub, da[0], db[0]);
  ok[1] = lane_entry<C, 1>(sub, da[1], db[1]);
  ok[2] = lane_entry<C, 2>(sub, da[2], db[2]);
  ok[3] = lane_entry<C, 3>(sub, da[3], db[3]);
  ok[4] = lane_entry<C, 4>(sub, da[4], db[4]);
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    int m = n + da[q] + A * db[q];
    if (bb + db[q] < 0) m += N;
    if (bb + db[q] >= B) m -= N;
    // outside the annulus (zero block), or past the last entry of the row: no contribution
    nb[q] = ok[q] && a + da[q] >= 0 && a + da[q] < A ? m : -1;
  }
  const NodeInv<T> di(dinv, n);
  T c1 = (T)0, c2 = (T)0;
  if (MODE == ST_FIRST_X) c2 = (T)ld_early(coef);
  constexpr bool kStep = MODE == ST_STEP || MODE == ST_STEP_X || MODE == ST_STEP_RZ;
  if (kStep) { c1 = (T)ld_early(coef); c2 = (T)ld_early(coef + 1); }
  grid_dep_sync();
  const X2* v2 = reinterpret_cast<const X2*>(v);
  X2 vn[PER];
#pragma unroll
  for (int q = 0; q < PER; ++q) vn[q] = v2[nb[q] < 0 ? n : nb[q]];
  const X2 own = v2[n];
  const X2 rv = reinterpret_cast<const X2*>(MODE == ST_FIRST_X ? b : r)[n];
  X2 xv;
  xv.x = xv.y = (T)0;
  double2 rrv = make_double2(0.0, 0.0);
  if (MODE == ST_STEP_RZ) rrv = reinterpret_cast<const double2*>(rr)[n];
  if (kStep) xv = reinterpret_cast<const X2*>(x)[n];
  T s0 = (T)0, s1 = (T)0;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    if (nb[q] >= 0) {
      s0 += k[q].k00 * vn[q].x + k[q].k01 * vn[q].y;
      s1 += k[q].k10 * vn[q].x + k[q].k11 * vn[q].y;
    }
  }
#pragma unroll
  for (int o = NPW; o < 32; o <<= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
  }
  if (!live || sub != 0) return 0.0;
  X2 rn;
  rn.x = rv.x - s0;
  rn.y = rv.y - s1;
  reinterpret_cast<X2*>(r)[n] = rn;
  if (MODE == ST_RESIDUAL) return 0.0;
  T z0, z1;
  di.apply(rn.x, rn.y, z0, z1);
  X2 dn;
  if (MODE == ST_FIRST_X) {
    dn.x = c2 * z0;
    dn.y = c2 * z1;
  } else {
    dn.x = c1 * own.x + c2 * z0;
    dn.y = c1 * own.y + c2 * z1;
    if (MODE == ST_STEP_X) {
      xv.x += own.x;
      xv.y += own.y;
    }
    xv.x += dn.x;
    xv.y += dn.y;
    reinterpret_cast<X2*>(x)[n] = xv;
  }
  if (MODE == ST_STEP_RZ) return rrv.x * (double)xv.x + rrv.y * (double)xv.y;   // nobody reads d again
  reinterpret_cast<X2*>(d)[n] = dn;
  return 0.0;
}

// CTAs [0, nb0) take class 0, the next nb1 class 1, and so on.
constexpr int kStThreads = 128;
template <int MODE, typename T>
__global__ void __launch_bounds__(kStThreads) k_stencil_step(const T* __restrict__ S, const T* v, const T* b, T* r,
                                                             T* x, T* d, const T* __restrict__ dinv,
                                                             const double* __restrict__ coef, int ncr, int nct,
                                                             int nb0, int nb1, int nb2, RzOut rz) {
  grid_dep_launch();
  int blk = blockIdx.x;
  double s;
  if (blk < nb0) {
    s = smooth_node<0, MODE, T>(S, v, b, r, x, d, dinv, coef, blk, ncr, nct, rz.r);
  } else if ((blk -= nb0) < nb1) {
    s = smooth_node<1, MODE, T>(S, v, b, r, x, d, dinv, coef, blk, ncr, nct, rz.r);
  } else if ((blk -= nb1) < nb2) {
    s = smooth_node<2, MODE, T>(S, v, b, r, x, d, dinv, coef, blk, ncr, nct, rz.r);
  } else {
    s = smooth_node<3, MODE, T>(S, v, b, r, x, d, dinv, coef, blk - nb2, ncr, nct, rz.r);
  }
  if (MODE == ST_STEP_RZ) block_add(rz.yy ? sqrt(*rz.yy) * s : s, rz.out);
}

template <int MODE, typename T>
static void launch_stencil_step(const Level& g, const T* S, const T* v, const T* b, T* r, T* x, T* d, const T* dinv,
                                const double* coef, cudaStream_t s, const RzOut& rz = RzOut()) {
  int nb[4];
  for (int c = 0; c < 4; ++c)
    nb[c] = (int)div_up((int64_t)st_nodes(c, g.ncr, g.nct) * st_lanes(c), kStThreads);
  klaunch(k_stencil_step<MODE, T>, nb[0] + nb[1] + nb[2] + nb[3], kStThreads, 0, s, S, v, b, r, x, d, dinv, coef,
          g.ncr, g.nct, nb[0], nb[1], nb[2], rz);
}

template <typename T>
static void launch_stencil_assemble(const Level& g, const T* K, T* S, cudaStream_t s) {
  klaunch(k_stencil_assemble<T>, dim3((unsigned)div_up(st_nodes(0, g.ncr, g.nct), 128), 4), 128, 0, s, K, S, g.ncr,
          g.nct);
  DP_LAUNCH_CHECK();
}

}  // namespace dp
