// Geometric multigrid preconditioner for the velocity block K (free DOFs).
//
// The reference inverts K[ifree, ifree] with a sparse LU once per solve and
// back-substitutes per outer iteration (src/PardisoSolvers.jl:247-256,
// :274-278).  On the device the inner solve is PCG preconditioned by one
// V-cycle of this hierarchy.
//
// Hierarchy.  The split-1 annulus with (ncr, nct) cells is nested in the one
// with (ncr/2, nct/2) cells: every coarse triangle is the union of 4 fine
// triangles and the fine diagonals continue the coarse ones, so coarse P2 is a
// subspace of fine P2 in (theta, r).  Prolongation P interpolates each polar
// component with the coarse P2 basis.  Coarse operators are Galerkin,
// A_c = P^T A P, computed element by element: K_E = sum_{children f}
// P_f^T K_f P_f with the 6x6 local interpolation P_f of each child position,
// followed by the coarse free-slip mask.  This keeps every level in the same
// packed element-by-element form as the fine level.
// Smoother: Chebyshev polynomial in D^-1 A (point Jacobi), bounds from a
// 10-step CG-Lanczos estimate of lambda_max.  Coarsest level: assembled densely,
// inverted once per setup by block Gauss-Jordan (32 pivots per panel) and
// applied as a dense mat-vec.
#include <algorithm>
#include <cmath>
#include <stdexcept>

#include "kernels.cuh"
#include "mg.cuh"

namespace dp {

// ---- host-side constant tables ---------------------------------------------
struct ChildTable {
  int dr[2][4], dt[2][4], tf[2][4];  // child cell offset (radial, angular) and type
  double P[2][4][6][6];              // P[coarse type][child][fine local][coarse local]
};
__constant__ ChildTable c_child;

static void p2_values(double xi, double eta, double N[6]) {
  const double t = 1.0 - xi - eta;
  N[0] = t * (2.0 * t - 1.0);
  N[1] = xi * (2.0 * xi - 1.0);
  N[2] = eta * (2.0 * eta - 1.0);
  N[3] = 4.0 * xi * t;
  N[4] = 4.0 * xi * eta;
  N[5] = 4.0 * eta * t;
}

// Local node offsets (radial a, angular b) of the 6 nodes of a triangle of type t
// inside its cell, in units of the P2 lattice of that level.
static const int kLocA[2][6] = {{0, 0, 2, 0, 1, 1}, {0, 2, 2, 1, 2, 1}};
static const int kLocB[2][6] = {{0, 2, 0, 1, 1, 0}, {2, 2, 0, 2, 1, 1}};

// Coarse reference coordinates of a point given in fine-lattice offsets
// (alpha radial, beta angular) from the coarse cell origin (coarse cell = 4x4).
static void coarse_ref(int type, double alpha, double beta, double* xi, double* eta) {
  if (type == 0) {  // v1 (0,0), v2 (0,4), v3 (4,0): point = (4 eta, 4 xi)
    *xi = beta / 4.0;
    *eta = alpha / 4.0;
  } else {          // v1 (0,4), v2 (4,4), v3 (4,0): point = (4 xi + 4 eta, 4 - 4 eta)
    *eta = (4.0 - beta) / 4.0;
    *xi = (alpha + beta - 4.0) / 4.0;
  }
}

// Restriction stencils.  R = P^T is translation invariant on the structured
// lattice: the fine nodes inside the support of a coarse basis function, and
// their weights, depend only on the parity class (a_c mod 2, b_c mod 2) of the
// coarse node.  The table is built once from the prolongation rule on an
// interior node of each class; at the walls the fine nodes outside the annulus
// are simply absent.  This turns the restriction into a gather (no atomics,
// no zeroing pass, deterministic).
constexpr int kRMax = 64;
constexpr int kRTaps = 25;  // largest stencil (vertex class)
struct RestrictTable {
  int n[4];
  signed char da[4][kRMax], db[4][kRMax];
  double w[4][kRMax];
};
__constant__ RestrictTable c_rtab;

static void host_fine_weights(int a, int b, int ncrc, int Ac, int Bc, int cn[6], double w[6]) {
  int IR = a >> 2;
  if (IR >= ncrc) IR = ncrc - 1;
  const int IT = b >> 2;
  const int alpha = a - 4 * IR, beta = b - 4 * IT;
  const int ct = (alpha + beta <= 4) ? 0 : 1;
  double xi, eta;
  coarse_ref(ct, alpha, beta, &xi, &eta);
  p2_values(xi, eta, w);
  for (int k = 0; k < 6; ++k) {
    const int ac = 2 * IR + kLocA[ct][k];
    int bc = 2 * IT + kLocB[ct][k];
    if (bc >= Bc) bc -= Bc;
    cn[k] = ac + Ac * bc;
  }
}

static void upload_restriction_table() {
  RestrictTable R{};
  const int ncrc = 8, nctc = 16, Ac = 2 * ncrc + 1, Bc = 2 * nctc, Af = 4 * ncrc + 1, Bf = 4 * nctc;
  for (int cls = 0; cls < 4; ++cls) {
    const int ac = 8 + (cls & 1), bc = 12 + (cls >> 1);
    const int target = ac + Ac * bc;
    int m = 0;
    for (int da = -4; da <= 4; ++da)
      for (int db = -4; db <= 4; ++db) {
        const int a = 2 * ac + da, b = 2 * bc + db;
        if (a < 0 || a >= Af || b < 0 || b >= Bf) continue;
        int cn[6];
        double w[6];
        host_fine_weights(a, b, ncrc, Ac, Bc, cn, w);
        double wt = 0.0;
        for (int k = 0; k < 6; ++k)
          if (cn[k] == target) wt += w[k];
        if (wt != 0.0) {
          if (m >= kRMax) throw std::runtime_error("restriction table overflow");
          R.da[cls][m] = (signed char)da;
          R.db[cls][m] = (signed char)db;
          R.w[cls][m] = wt;
          ++m;
        }
      }
    if (m > kRTaps) throw std::runtime_error("restriction stencil larger than expected");
    R.n[cls] = m;
  }
  DP_CUDA(cudaMemcpyToSymbol(c_rtab, &R, sizeof(R)));
}

void upload_mg_constants() {
  ChildTable T{};
  // coarse A children: (0,0,A) (0,0,B) (0,1,A) (1,0,A); coarse B: (0,1,B) (1,0,B) (1,1,A) (1,1,B)
  const int dr[2][4] = {{0, 0, 0, 1}, {0, 1, 1, 1}};
  const int dt[2][4] = {{0, 0, 1, 0}, {1, 0, 1, 1}};
  const int tf[2][4] = {{0, 1, 0, 0}, {1, 1, 0, 1}};
  for (int ct = 0; ct < 2; ++ct)
    for (int ch = 0; ch < 4; ++ch) {
      T.dr[ct][ch] = dr[ct][ch];
      T.dt[ct][ch] = dt[ct][ch];
      T.tf[ct][ch] = tf[ct][ch];
      for (int i = 0; i < 6; ++i) {
        const double alpha = 2 * dr[ct][ch] + kLocA[tf[ct][ch]][i];
        const double beta = 2 * dt[ct][ch] + kLocB[tf[ct][ch]][i];
        double xi, eta, N[6];
        coarse_ref(ct, alpha, beta, &xi, &eta);
        p2_values(xi, eta, N);
        for (int k = 0; k < 6; ++k) T.P[ct][ch][i][k] = N[k];
      }
    }
  DP_CUDA(cudaMemcpyToSymbol(c_child, &T, sizeof(T)));
  upload_restriction_table();
}

// ---- Galerkin coarsening ---------------------------------------------------------
// K_E = sum over the 4 children of P_f^T K_f P_f, sums in FP64.  A CTA takes 32
// consecutive coarse cells: the 8 fine elements of each are copied to shared
// memory once (coalesced, 16-byte groups as they are stored), then each of the
// 12 warps owns one (coarse type, coarse node l), its lanes the 32 cells: the
// two columns of node l of K_f P are summed over the packed entries with the
// 6 weights P[.][l] in registers, then P^T is applied to them.  The coarse
// elements leave through shared memory as coalesced 16-byte groups.
// Bound by FP64 FMA and FP32 -> FP64 conversion (6.9 k FMA a coarse element).
// The form it replaces, a thread per (coarse element, entry), re-read each
// child entry ~36 times: 10.55 ms for the first coarsening at 512x4096.
template <typename T>
struct GalerkinTile {
  static constexpr int kVec = KVec<T>::n;            // 16-byte groups per element
  static constexpr int kPer = 16 / sizeof(T);
  static constexpr int kSlot = kVec * 32 + 2;        // groups per fine slot; +2 keeps the copy free of bank conflicts
  static constexpr size_t kSmem = 16 * (size_t)(8 * kSlot + 2 * kVec * 32);
};
constexpr int kGalThreads = 384;   // 12 warps: (type, node)

template <typename T>
__global__ void __launch_bounds__(kGalThreads) k_galerkin(const T* __restrict__ Kf, T* __restrict__ Kc, int ncrc,
                                                          int nctc, int ncrf, int pin) {
  typedef GalerkinTile<T> G;
  typedef typename KVec<T>::V VT;
  grid_dep_wait();
  extern __shared__ __align__(16) unsigned char gal_raw[];
  VT* in = reinterpret_cast<VT*>(gal_raw);          // [fine slot 4 dt + 2 dr + tf][group][cell]
  VT* out = in + 8 * G::kSlot;                      // [type][group][cell]
  const int ncell = ncrc * nctc, q0 = blockIdx.x * 32;
  for (int idx = threadIdx.x; idx < 8 * 32 * G::kVec; idx += kGalThreads) {
    const int el4 = idx & 127, rest = idx >> 7;      // 4 consecutive fine elements per cell and angular row
    const int j = rest % G::kVec, dt = rest / G::kVec;
    const int cell = el4 >> 2, Q = q0 + cell;
    if (Q < ncell) {
      const int IR = Q % ncrc, IT = Q / ncrc;
      const int64_t e = 4 * (int64_t)IR + (el4 & 3) + 2 * (int64_t)ncrf * (2 * IT + dt);
      in[(4 * dt + (el4 & 3)) * G::kSlot + j * 32 + cell] =
          reinterpret_cast<const VT*>(Kf)[(e >> 5) * (32 * G::kVec) + j * 32 + (e & 31)];
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int ct = w / 6, l = w - 6 * ct;
  const int Q = q0 + lane;
  if (Q < ncell) {
    double acc[6][2][2];
#pragma unroll
    for (int k = 0; k < 6; ++k) acc[k][0][0] = acc[k][0][1] = acc[k][1][0] = acc[k][1][1] = 0.0;
#pragma unroll 1
    for (int ch = 0; ch < 4; ++ch) {
      const VT* src = in + (4 * c_child.dt[ct][ch] + 2 * c_child.dr[ct][ch] + c_child.tf[ct][ch]) * G::kSlot + lane;
      double wl[6], s[6][2][2];   // wl = P[.][l]; s[i] = the 2x2 block (row node i, column node l) of K_f P
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        wl[i] = c_child.P[ct][ch][i][l];
        s[i][0][0] = s[i][0][1] = s[i][1][0] = s[i][1][1] = 0.0;
      }
#pragma unroll
      for (int C = 0; C < 12; ++C) {
#pragma unroll
        for (int R = C; R < 12; ++R) {
          const int p = packed_index12(R, C);
          T kk[G::kPer];
          vec_to(src[(p / G::kPer) * 32], kk);
          const double v = (double)kk[p % G::kPer];
          s[R >> 1][R & 1][C & 1] += v * wl[C >> 1];
          if (R != C) s[C >> 1][C & 1][R & 1] += v * wl[R >> 1];
        }
      }
#pragma unroll
      for (int k = 0; k < 6; ++k) {
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          const double pik = c_child.P[ct][ch][i][k];
          if (pik == 0.0) continue;   // the same for the whole warp
          acc[k][0][0] += pik * s[i][0][0];
          acc[k][0][1] += pik * s[i][0][1];
          acc[k][1][0] += pik * s[i][1][0];
          acc[k][1][1] += pik * s[i][1][1];
        }
      }
    }
    // coarse constraint mask (free slip + optional tangential pin)
    const int IR = Q % ncrc, IT = Q / ncrc, Bc = 2 * nctc, amax = 2 * ncrc;
    auto fixed = [&](int k, int comp) {
      int b = 2 * IT + kLocB_dev(ct, k);
      if (b >= Bc) b -= Bc;
      return dof_fixed(2 * IR + kLocA_dev(ct, k), b, comp, amax, pin);
    };
    T* o = reinterpret_cast<T*>(out + (size_t)ct * G::kVec * 32 + lane);
    const bool fl[2] = {fixed(l, 0), fixed(l, 1)};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      if (k < l) continue;
      const bool fk[2] = {fixed(k, 0), fixed(k, 1)};
#pragma unroll
      for (int al = 0; al < 2; ++al) {
#pragma unroll
        for (int be = 0; be < 2; ++be) {
          if (k == l && al < be) continue;
          const int p = packed_index12(2 * k + al, 2 * l + be);
          o[(size_t)(p / G::kPer) * 32 * G::kPer + p % G::kPer] = (T)(fk[al] || fl[be] ? 0.0 : acc[k][al][be]);
        }
      }
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < 2 * 32 * G::kVec; idx += kGalThreads) {
    const int el2 = idx & 63, j = idx >> 6, cell = el2 >> 1;
    if (q0 + cell < ncell) {
      const int64_t E = 2 * (int64_t)q0 + el2;
      reinterpret_cast<VT*>(Kc)[(E >> 5) * (32 * G::kVec) + j * 32 + (E & 31)] =
          out[(el2 & 1) * G::kVec * 32 + j * 32 + cell];
    }
  }
}

// ---- nodal 2x2 diagonal blocks and their inverses ----------------------------
// Per node: the sum of its 2x2 diagonal blocks over the elements that hold it (a
// gather in a fixed order, no atomics and no buffer of sums) and the inverse of
// that block (block = 1) or of its diagonal (block = 0).  Constrained DOFs get
// zero rows/columns so the smoother never touches them.  One thread per 2x2
// node block, one node of each parity class, as in k_node_gather.
template <int PA, int PB, typename T>
__device__ __forceinline__ void diag_invert_node(const T* __restrict__ K, T* __restrict__ dinv, int i, int j, int ncr,
                                                 int nct, int pin, int block) {
  const int a = 2 * i + PA, b = 2 * j + PB;
  if (a > 2 * ncr) return;
  double d00 = 0.0, d01 = 0.0, d11 = 0.0;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      if ((loc_a(t, k) & 1) != PA || (loc_b(t, k) & 1) != PB) continue;   // resolved at compile time
      const int ir = i + ((PA - loc_a(t, k)) >> 1);
      int it = j + ((PB - loc_b(t, k)) >> 1);
      if (ir < 0 || ir >= ncr) continue;
      if (it < 0) it += nct;
      const int64_t e = 2 * ((int64_t)ir + (int64_t)ncr * it) + t;
      d00 += (double)K[kidx<T>(packed_index12(2 * k, 2 * k), e)];
      d01 += (double)K[kidx<T>(packed_index12(2 * k + 1, 2 * k), e)];
      d11 += (double)K[kidx<T>(packed_index12(2 * k + 1, 2 * k + 1), e)];
    }
  }
  const bool f0 = dof_fixed(a, b, 0, 2 * ncr, pin), f1 = dof_fixed(a, b, 1, 2 * ncr, pin);
  if (!block) d01 = 0.0;
  double i00 = 0.0, i01 = 0.0, i11 = 0.0;
  const double det = d00 * d11 - d01 * d01;
  if (f0 || f1 || d01 == 0.0 || !(det > 0.0)) {
    i00 = (!f0 && d00 > 0.0) ? 1.0 / d00 : 0.0;
    i11 = (!f1 && d11 > 0.0) ? 1.0 / d11 : 0.0;
  } else {
    i00 = d11 / det;
    i01 = -d01 / det;
    i11 = d00 / det;
  }
  T* o = dinv + 3 * (a + (int64_t)(2 * ncr + 1) * b);
  o[0] = (T)i00;
  o[1] = (T)i01;
  o[2] = (T)i11;
}

template <typename T>
__global__ void __launch_bounds__(256) k_diag_invert(const T* __restrict__ K, T* __restrict__ dinv, int ncr, int nct,
                                                     int pin, int block) {
  grid_dep_wait();
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= (int64_t)(ncr + 1) * nct) return;
  const int j = (int)(q / (ncr + 1)), i = (int)(q - (int64_t)j * (ncr + 1));
  diag_invert_node<0, 0, T>(K, dinv, i, j, ncr, nct, pin, block);
  diag_invert_node<1, 0, T>(K, dinv, i, j, ncr, nct, pin, block);
  diag_invert_node<0, 1, T>(K, dinv, i, j, ncr, nct, pin, block);
  diag_invert_node<1, 1, T>(K, dinv, i, j, ncr, nct, pin, block);
}

template <typename T>
__device__ inline void bj_apply(const T* __restrict__ dinv, int64_t n, double r0, double r1, double& z0, double& z1) {
  const double a = (double)dinv[3 * n], b = (double)dinv[3 * n + 1], c = (double)dinv[3 * n + 2];
  z0 = a * r0 + b * r1;
  z1 = b * r0 + c * r1;
}

// ---- transfers ---------------------------------------------------------------
// Fine node (a, b) -> containing coarse element and the 6 coarse P2 weights.
__device__ inline void fine_node_weights(int a, int b, int ncrc, int Ac, int Bc, int cn[6], double w[6]) {
  int IR = a >> 2;
  if (IR >= ncrc) IR = ncrc - 1;
  const int IT = b >> 2;
  const int alpha = a - 4 * IR, beta = b - 4 * IT;
  const int ct = (alpha + beta <= 4) ? 0 : 1;
  double xi, eta;
  if (ct == 0) { xi = beta * 0.25; eta = alpha * 0.25; }
  else { eta = (4 - beta) * 0.25; xi = (alpha + beta - 4) * 0.25; }
  const double t = 1.0 - xi - eta;
  w[0] = t * (2.0 * t - 1.0);
  w[1] = xi * (2.0 * xi - 1.0);
  w[2] = eta * (2.0 * eta - 1.0);
  w[3] = 4.0 * xi * t;
  w[4] = 4.0 * xi * eta;
  w[5] = 4.0 * eta * t;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int ac = 2 * IR + kLocA_dev(ct, k);
    int bc = 2 * IT + kLocB_dev(ct, k);
    if (bc >= Bc) bc -= Bc;
    cn[k] = ac + Ac * bc;
  }
}

}  // namespace dp
#include "halo.cu"
namespace dp {

// xf += P xc (per fine node, gather); also sets rf = bf (the fine level's
// residual buffer, from which the next apply subtracts A xf) unless rf is null.
// d1 (and d2) given: xf holds the last step of the pre-smoothing only, and the
// smoothed x is (d1 + d2) + xf.
template <typename T>
__global__ void k_prolong_add(const T* xc, T* xf, const T* d1, const T* d2, const T* bf,
                              T* rf, int Af, int Bf, int ncrc, int Ac, int Bc, int pin) {
  grid_dep_launch();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= Af * Bf) return;
  const int b = n / Af, a = n - b * Af;
  int cn[6];
  double w[6];
  fine_node_weights(a, b, ncrc, Ac, Bc, cn, w);
  grid_dep_sync();
  // the 6 nodes of the containing coarse element are always valid: gather them
  // all unconditionally (zero weights included) so the loads issue together
  typedef typename V2<T>::T X2;
  const X2* xc2 = reinterpret_cast<const X2*>(xc);
  X2 v[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) v[k] = xc2[cn[k]];
  X2 xv = reinterpret_cast<const X2*>(xf)[n];
  if (d1) {
    X2 u = reinterpret_cast<const X2*>(d1)[n];
    if (d2) {
      const X2 w2 = reinterpret_cast<const X2*>(d2)[n];
      u.x += w2.x;
      u.y += w2.y;
    }
    xv.x = u.x + xv.x;
    xv.y = u.y + xv.y;
  }
  X2 bv = xv;
  if (rf) bv = reinterpret_cast<const X2*>(bf)[n];
  T s0 = (T)0, s1 = (T)0;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    s0 += (T)w[k] * v[k].x;
    s1 += (T)w[k] * v[k].y;
  }
  if (!dof_fixed(a, b, 0, Af - 1, pin)) xv.x += s0;
  if (!dof_fixed(a, b, 1, Af - 1, pin)) xv.y += s1;
  reinterpret_cast<X2*>(xf)[n] = xv;
  if (rf) reinterpret_cast<X2*>(rf)[n] = bv;
}

// bc = P^T r per coarse node (gather over the class stencil); constrained DOFs
// of either level are excluded.  blockIdx.y is the parity class.  Four lanes
// gather for one coarse node, at most 7 taps each, and add up by shuffles.
// The gather is a chain of two short latencies behind a launch; what took most
// of it was the table (each lane of four reads its own entry of constant
// memory, so a read is four), which now happens before the wait together with
// D^-1: an inner iteration with 2 (16x128) to 3 (32x256) of these launches takes
// 56.9 and 78.3 us instead of 59.2 and 81.1 (including the same for the
// weights in k_halo_up).
// first != 0 also takes the coarse level's first Chebyshev step from x = 0
// (the work of k_cheb_first): rc = bc, dc = xc = coef[0] D^-1 bc (no xc if it is
// null), and tc = 0 when tc is given (the cluster tail's levels accumulate into t).
template <typename T>
__global__ void __launch_bounds__(256) k_restrict_g(const T* r, T* bc, int Af, int Bf, int Ac, int Bc, int pin,
                                                    int first, const T* dinv_c, T* xc, T* rc, T* dc, T* tc,
                                                    const double* coef_c) {
  grid_dep_launch();
  constexpr int LPN = 4, PER = (kRTaps + LPN - 1) / LPN;
  const int cls = blockIdx.y;
  const int pa = cls & 1, pb = cls >> 1;
  const int nA = (Ac - pa + 1) >> 1;  // coarse a = pa, pa + 2, ... <= Ac - 1
  const int gidx = blockIdx.x * blockDim.x + threadIdx.x;
  const int idx = gidx / LPN, sub = gidx % LPN;
  const bool live = idx < nA * (Bc >> 1);
  const int ac = live ? 2 * (idx % nA) + pa : pa, bcn = live ? 2 * (idx / nA) + pb : pb;
  const int n = ac + Ac * bcn;
  typedef typename V2<T>::T X2;
  const int m = live ? c_rtab.n[cls] : 0;
  int f[PER];
  float w0[PER], w1[PER];   // dyadic fractions, exact in FP32
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int j = sub + LPN * q, jj = j < m ? j : 0;
    const int a = 2 * ac + c_rtab.da[cls][jj];
    int b = 2 * bcn + c_rtab.db[cls][jj];
    b += (b < 0) ? Bf : 0;
    b -= (b >= Bf) ? Bf : 0;
    const bool in = j < m && a >= 0 && a < Af;
    const float w = (float)c_rtab.w[cls][jj];
    f[q] = in ? a + Af * b : -1;
    w0[q] = dof_fixed(a, b, 0, Af - 1, pin) ? 0.f : w;
    w1[q] = dof_fixed(a, b, 1, Af - 1, pin) ? 0.f : w;
  }
  T da = (T)0, db = (T)0, dd = (T)0;
  double it = 0.0;
  if (first) {
    da = ld_early(dinv_c + 3 * (int64_t)n);
    db = ld_early(dinv_c + 3 * (int64_t)n + 1);
    dd = ld_early(dinv_c + 3 * (int64_t)n + 2);
    it = ld_early(coef_c);
  }
  grid_dep_sync();
  const X2* r2 = reinterpret_cast<const X2*>(r);
  X2 rv[PER];
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    rv[q].x = rv[q].y = (T)0;
    if (f[q] >= 0) rv[q] = r2[f[q]];
  }
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    s0 += (double)w0[q] * (double)rv[q].x;
    s1 += (double)w1[q] * (double)rv[q].y;
  }
  // every lane of the warp takes part in the shuffles (dead lanes add zeros)
#pragma unroll
  for (int o = 1; o < LPN; o <<= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
  }
  if (!live || sub != 0) return;
  X2 v;
  const double b0 = dof_fixed(ac, bcn, 0, Ac - 1, pin) ? 0.0 : s0;
  const double b1 = dof_fixed(ac, bcn, 1, Ac - 1, pin) ? 0.0 : s1;
  v.x = (T)b0;
  v.y = (T)b1;
  reinterpret_cast<X2*>(bc)[n] = v;
  if (first) {
    reinterpret_cast<X2*>(rc)[n] = v;
    v.x = (T)(it * ((double)da * b0 + (double)db * b1));
    v.y = (T)(it * ((double)db * b0 + (double)dd * b1));
    reinterpret_cast<X2*>(dc)[n] = v;
    if (xc) reinterpret_cast<X2*>(xc)[n] = v;
    if (tc) {
      v.x = v.y = (T)0;
      reinterpret_cast<X2*>(tc)[n] = v;
    }
  }
}

// Tiled form of the same restriction for the large levels.  One CTA = 16 x 16
// coarse nodes; the fine values r of the CTA's stencil footprint (a 39 x 39
// patch of fine nodes, constrained fine DOFs zeroed) are read from global
// memory once into shared memory, and each coarse node gathers its class
// stencil from there (the gather form reads every fine value ~4 times through
// L2).  Warps are class-uniform (64 coarse nodes of each parity class), so the
// stencil table reads are constant-cache broadcasts.  Arithmetic in the level's
// precision (the stencil weights are dyadic fractions, exact in FP32).
constexpr int kRTile = 16;
constexpr int kRPatch = 2 * (kRTile - 1) + 1 + 8;   // 39: stencil offsets reach 4 fine nodes each way
// Patch node (la, lb) in shared memory: the radial index split into 4 planes, so
// that the 8 coarse nodes of a lane group (4 fine nodes apart) are neighbours, and
// a pitch that moves the warp's next group (4 rows on) by half of the banks
// (FP32): 2 wavefronts per read instead of 8.  With the fill's loads all in
// flight and D^-1 before the wait, an inner iteration takes 113 instead of 116.5
// us at 64x512, 239.6 instead of 246 at 128x1024 and 698 instead of 706 at
// 256x2048.
constexpr int kRPitch = 42;
__device__ __forceinline__ int rpatch_at(int la, int lb) { return lb * kRPitch + (la & 3) * 10 + (la >> 2); }
template <typename T>
__global__ void __launch_bounds__(256) k_restrict_tile(const T* r, T* bc, int Af, int Bf, int Ac, int Bc, int pin,
                                                       int first, const T* dinv_c, T* xc, T* rc, T* dc, T* tc,
                                                       const double* coef_c) {
  grid_dep_launch();
  typedef typename V2<T>::T X2;
  __shared__ X2 sp[kRPatch * kRPitch];
  const int ac0 = blockIdx.x * kRTile, bc0 = blockIdx.y * kRTile;
  const int fa0 = 2 * ac0 - 4, fb0 = 2 * bc0 - 4;
  const int cls = threadIdx.x >> 6, loc = threadIdx.x & 63;
  const int pa = cls & 1, pb = cls >> 1;
  const int ac = ac0 + 2 * (loc & 7) + pa, bcn = bc0 + 2 * (loc >> 3) + pb;
  const bool live = ac < Ac && bcn < Bc;
  const int n = live ? ac + Ac * bcn : 0;
  T da = (T)0, db = (T)0, dd = (T)0, it = (T)0;
  if (first) {
    da = ld_early(dinv_c + 3 * (int64_t)n);
    db = ld_early(dinv_c + 3 * (int64_t)n + 1);
    dd = ld_early(dinv_c + 3 * (int64_t)n + 2);
    it = (T)ld_early(coef_c);
  }
  grid_dep_sync();
  const X2* r2 = reinterpret_cast<const X2*>(r);
  constexpr int kFill = (kRPatch * kRPatch + 255) / 256;
  X2 v[kFill];
#pragma unroll
  for (int q = 0; q < kFill; ++q) {          // all loads in flight, then the stores
    const int k = threadIdx.x + 256 * q, la = k % kRPatch, lb = k / kRPatch;
    const int a = fa0 + la;
    int b = fb0 + lb;
    b += (b < 0) ? Bf : 0;                   // the patch reaches at most 4 nodes past either end
    b -= (b >= Bf) ? Bf : 0;
    v[q].x = v[q].y = (T)0;
    if (lb < kRPatch && a >= 0 && a < Af) {
      v[q] = r2[a + (int64_t)Af * b];
      if (dof_fixed(a, b, 0, Af - 1, pin)) v[q].x = (T)0;
      if (dof_fixed(a, b, 1, Af - 1, pin)) v[q].y = (T)0;
    }
  }
#pragma unroll
  for (int q = 0; q < kFill; ++q) {
    const int k = threadIdx.x + 256 * q;
    if (k < kRPatch * kRPatch) sp[rpatch_at(k % kRPatch, k / kRPatch)] = v[q];
  }
  __syncthreads();
  if (!live) return;
  const int m = c_rtab.n[cls];
  T s0 = (T)0, s1 = (T)0;
#pragma unroll 5
  for (int j = 0; j < m; ++j) {
    const int la = 2 * (ac - ac0) + 4 + c_rtab.da[cls][j];
    const int lb = 2 * (bcn - bc0) + 4 + c_rtab.db[cls][j];
    const X2 u = sp[rpatch_at(la, lb)];
    const T w = (T)c_rtab.w[cls][j];
    s0 += w * u.x;
    s1 += w * u.y;
  }
  const T b0 = dof_fixed(ac, bcn, 0, Ac - 1, pin) ? (T)0 : s0;
  const T b1 = dof_fixed(ac, bcn, 1, Ac - 1, pin) ? (T)0 : s1;
  X2 bv;
  bv.x = b0;
  bv.y = b1;
  reinterpret_cast<X2*>(bc)[n] = bv;
  if (first) {
    const T z0 = da * b0 + db * b1;
    const T z1 = db * b0 + dd * b1;
    X2 dv;
    dv.x = it * z0;
    dv.y = it * z1;
    if (tc) {
      X2 zero;
      zero.x = (T)0;
      zero.y = (T)0;
      reinterpret_cast<X2*>(tc)[n] = zero;
    }
    reinterpret_cast<X2*>(rc)[n] = bv;
    reinterpret_cast<X2*>(dc)[n] = dv;
    if (xc) reinterpret_cast<X2*>(xc)[n] = dv;
  }
}

// ---- Chebyshev smoother vector steps (per node, coefficients read from device) --
// The residual r lives in one buffer that the applies between the steps update
// in place (r -= A d, launch_apply_K_sub).  With 2 or 3 steps (the default 3)
// the steps only form the d_k, each in a buffer of its own, and x is put
// together where it is next needed anyway: by the prolongation after the
// pre-smoothing (whose last d lies in x) and by the last post-smoothing step.
// That moves 272 instead of 328 bytes per FP32 node and V-cycle: the FP32
// V-cycle takes 2250 instead of 2330 us at 512x4096 and 174 instead of 186 at
// 64x512, within 1 % of the same at 128x1024.
// The kernels compute in the precision of the level (FP32 on the FP32
// hierarchy) and move each node's pair of components with one 8/16-byte
// access, all loads issued before the arithmetic.

// first step from x = 0: r = b, d = (1/theta) D^-1 b (x = d unless x is null)
template <typename T>
__global__ void k_cheb_first(const T* b, const T* __restrict__ dinv, T* x,
                             T* r, T* d, const double* __restrict__ coef, int64_t nnod) {
  grid_dep_launch();
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= nnod) return;
  typedef typename V2<T>::T X2;
  const NodeInv<T> di(dinv, n);
  const T it = (T)ld_early(coef);
  grid_dep_sync();
  const X2 bv = reinterpret_cast<const X2*>(b)[n];
  T z0, z1;
  di.apply(bv.x, bv.y, z0, z1);
  X2 dv;
  dv.x = it * z0; dv.y = it * z1;
  reinterpret_cast<X2*>(r)[n] = bv;
  reinterpret_cast<X2*>(d)[n] = dv;
  if (x) reinterpret_cast<X2*>(x)[n] = dv;
}
// first step from a given x (r = b - Ax on entry): d = (1/theta) D^-1 r (x += d unless x is null)
template <typename T>
__global__ void k_cheb_first_x(const T* r, const T* __restrict__ dinv, T* x,
                               T* d, const double* __restrict__ coef, int64_t nnod) {
  grid_dep_launch();
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= nnod) return;
  typedef typename V2<T>::T X2;
  const NodeInv<T> di(dinv, n);
  const T it = (T)ld_early(coef);
  grid_dep_sync();
  const X2 rv = reinterpret_cast<const X2*>(r)[n];
  X2 xv;
  if (x) xv = reinterpret_cast<const X2*>(x)[n];
  X2 dv;
  T z0, z1;
  di.apply(rv.x, rv.y, z0, z1);
  dv.x = it * z0; dv.y = it * z1;
  reinterpret_cast<X2*>(d)[n] = dv;
  if (!x) return;
  xv.x += dv.x; xv.y += dv.y;
  reinterpret_cast<X2*>(x)[n] = xv;
}
// d_new = c1 d + c2 D^-1 r  (c1, c2 = coef[0], coef[1]; r already holds r - A d)
// CH_IN_PLACE: d = d_new, x += d_new;  CH_NEXT: dn = d_new;
// CH_LAST: x = ((x + e) + d) + d_new, e the step before d (null: none)
enum ChebStep { CH_IN_PLACE, CH_NEXT, CH_LAST };
template <int MODE, typename T>
__global__ void k_cheb_step(const T* r, const T* __restrict__ dinv, T* x, T* d, T* dn, const T* e,
                            const double* __restrict__ coef, int64_t nnod) {
  grid_dep_launch();
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= nnod) return;
  typedef typename V2<T>::T X2;
  const NodeInv<T> di(dinv, n);
  const T c1 = (T)ld_early(coef), c2 = (T)ld_early(coef + 1);
  grid_dep_sync();
  const X2 rv = reinterpret_cast<const X2*>(r)[n];
  const X2 dv = reinterpret_cast<const X2*>(d)[n];
  X2 xv, ev;
  if (MODE != CH_NEXT) xv = reinterpret_cast<const X2*>(x)[n];
  if (MODE == CH_LAST && e) ev = reinterpret_cast<const X2*>(e)[n];
  X2 nv;
  T z0, z1;
  di.apply(rv.x, rv.y, z0, z1);
  nv.x = c1 * dv.x + c2 * z0; nv.y = c1 * dv.y + c2 * z1;
  if (MODE == CH_IN_PLACE) reinterpret_cast<X2*>(d)[n] = nv;
  if (MODE == CH_NEXT) {
    reinterpret_cast<X2*>(dn)[n] = nv;
    return;
  }
  if (MODE == CH_LAST) {
    if (e) { xv.x += ev.x; xv.y += ev.y; }
    xv.x += dv.x; xv.y += dv.y;
  }
  xv.x += nv.x; xv.y += nv.y;
  reinterpret_cast<X2*>(x)[n] = xv;
}
// z = D^-1 r (nodal blocks)
template <typename T>
__global__ void k_bj(const T* __restrict__ dinv, const T* r, T* z, int64_t nnod) {
  grid_dep_wait();
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= nnod) return;
  double z0, z1;
  bj_apply<T>(dinv, n, (double)r[2 * n], (double)r[2 * n + 1], z0, z1);
  z[2 * n] = (T)z0;
  z[2 * n + 1] = (T)z1;
}

// ---- coarse dense solve --------------------------------------------------------
// The dense matrix row by row from the elements around each node (the gather of
// the node stencils: every entry written once, in a fixed order).
template <int C, int J, typename T>
__device__ __forceinline__ void dense_entry(const T* __restrict__ K, double* D, int i, int ia, int jb, int ncr, int nct) {
  constexpr int DA = StencilEntry<C, J>::da, DB = StencilEntry<C, J>::db;
  const int A = 2 * ncr + 1, B = 2 * nct, a = 2 * ia + (C & 1), b = 2 * jb + (C >> 1);
  if (a + DA < 0 || a + DA >= A) return;
  double acc[4];
  stencil_sum<C, J, T>(K, ia, jb, ncr, nct, acc);
  int bm = b + DB;
  bm += bm < 0 ? B : (bm >= B ? -B : 0);
  const int64_t n = 2 * (int64_t)A * B, row = 2 * (a + (int64_t)A * b), col = 2 * (a + DA + (int64_t)A * bm);
#pragma unroll
  for (int q = 0; q < 4; ++q) D[(row + (q >> 1)) * n + col + (q & 1)] = acc[q];
}
template <int C, typename T, int... J>
__device__ __forceinline__ void dense_rows(const T* __restrict__ K, double* D, int i, int ncr, int nct,
                                           std::integer_sequence<int, J...>) {
  const int nA = (C & 1) ? ncr : ncr + 1;
  const int ia = i % nA, jb = i / nA;
  (dense_entry<C, J, T>(K, D, i, ia, jb, ncr, nct), ...);
}
template <typename T>
__global__ void __launch_bounds__(64) k_dense_assemble(const T* __restrict__ K, double* D, int ncr, int nct) {
  grid_dep_wait();
  const int c = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= st_nodes(c, ncr, nct)) return;
  if (c == 0) dense_rows<0, T>(K, D, i, ncr, nct, std::make_integer_sequence<int, st_entries(0)>{});
  else if (c == 1) dense_rows<1, T>(K, D, i, ncr, nct, std::make_integer_sequence<int, st_entries(1)>{});
  else if (c == 2) dense_rows<2, T>(K, D, i, ncr, nct, std::make_integer_sequence<int, st_entries(2)>{});
  else dense_rows<3, T>(K, D, i, ncr, nct, std::make_integer_sequence<int, st_entries(3)>{});
}

// Identity on the diagonal of fixed (all-zero) rows, so the matrix stays SPD.
__global__ void k_dense_fix_diag(double* __restrict__ D, int n) {
  grid_dep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && D[(size_t)i * n + i] == 0.0) D[(size_t)i * n + i] = 1.0;
}

// Block Gauss-Jordan inversion of the SPD coarsest matrix, one panel of up to
// kGJPanel pivots K = [k0, k0 + b) at a time (no pivoting: the pivot blocks of an
// SPD matrix are SPD).  With W = A_KK^-1 and T = A_{:,K} W, the panel step maps A
// (old) to B (new):
//   B_KK = W,   B_Kj = W A_Kj,   B_iK = -T_iK,   B_ij = A_ij - T_iK A_Kj
// (i, j outside K).  After all panels B = A^-1.  One launch per panel: a CTA
// forms T for its 64 rows, updates its 64x64 tile from the 32 pivot rows (all
// in shared memory) and, if the tile holds the next pivot block, inverts that
// for the next launch while the other tiles are still at work.
// At n = 1152 a panel took 47 us as three launches with every entry's 64
// operands read through L1.
constexpr int kGJPanel = 32;

__global__ void __launch_bounds__(kGJPanel * kGJPanel) k_gj_panel_inverse(const double* __restrict__ A,
                                                                          double* __restrict__ W, int n, int k0,
                                                                          int b) {
  grid_dep_wait();
  __shared__ double s[kGJPanel][kGJPanel + 1];
  const int r = threadIdx.y, c = threadIdx.x;
  s[r][c] = (r < b && c < b) ? A[(size_t)(k0 + r) * n + k0 + c] : (r == c ? 1.0 : 0.0);
  __syncthreads();
  for (int k = 0; k < b; ++k) {
    const double ip = 1.0 / s[k][k];
    const double akc = s[k][c], ark = s[r][k];
    __syncthreads();                       // every read of pivot row/column before any write
    double v;
    if (r == k) v = (c == k) ? ip : akc * ip;
    else if (c == k) v = -ark * ip;
    else v = s[r][c] - ark * akc * ip;
    s[r][c] = v;
    __syncthreads();
  }
  W[r * kGJPanel + c] = s[r][c];
}

constexpr int kGJTile = 64;
constexpr size_t kGJSmem = sizeof(double) * (kGJPanel * kGJPanel + 2 * kGJTile * (kGJPanel + 1) +
                                             kGJPanel * kGJTile + 2 * kGJPanel * (kGJPanel + 1));

__global__ void __launch_bounds__(256) k_gj_panel(const double* A, double* B, const double* W, double* Wn, int n,
                                                  int k0) {
  grid_dep_wait();
  extern __shared__ __align__(16) double gj[];
  double(*sw)[kGJPanel] = reinterpret_cast<double(*)[kGJPanel]>(gj);
  double(*sa)[kGJPanel + 1] = reinterpret_cast<double(*)[kGJPanel + 1]>(gj + kGJPanel * kGJPanel);
  double(*st)[kGJPanel + 1] = sa + kGJTile;
  double(*sb)[kGJTile] = reinterpret_cast<double(*)[kGJTile]>(&st[kGJTile][0]);
  double(*sp)[kGJPanel][kGJPanel + 1] = reinterpret_cast<double(*)[kGJPanel][kGJPanel + 1]>(&sb[kGJPanel][0]);
  const int i0 = blockIdx.y * kGJTile, j0 = blockIdx.x * kGJTile, b = min(kGJPanel, n - k0);
  for (int q = threadIdx.x; q < kGJPanel * kGJPanel; q += 256) sw[q / kGJPanel][q % kGJPanel] = W[q];
  for (int q = threadIdx.x; q < kGJTile * kGJPanel; q += 256) {
    const int r = q / kGJPanel, m = q % kGJPanel;
    sa[r][m] = (i0 + r < n && m < b) ? A[(size_t)(i0 + r) * n + k0 + m] : 0.0;
  }
  for (int q = threadIdx.x; q < kGJPanel * kGJTile; q += 256) {
    const int m = q / kGJTile, c = q % kGJTile;
    sb[m][c] = (j0 + c < n && m < b) ? A[(size_t)(k0 + m) * n + j0 + c] : 0.0;
  }
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double v[4][4];   // rows ty + 16 r, columns tx + 16 c of the tile; the rows of K start from zero
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = i0 + ty + 16 * r, j = j0 + tx + 16 * c;
      const bool ik = i >= k0 && i < k0 + b;
      v[r][c] = (i < n && j < n && !ik) ? A[(size_t)i * n + j] : 0.0;
    }
  __syncthreads();
  // T rows (-W for the rows of K, which turns the update below into W A_Kj)
  for (int q = threadIdx.x; q < kGJTile * kGJPanel; q += 256) {
    const int r = q / kGJPanel, m = q % kGJPanel, i = i0 + r;
    double t = 0.0;
    if (i >= k0 && i < k0 + b) {
      t = -sw[i - k0][m];
    } else {
#pragma unroll 8
      for (int l = 0; l < kGJPanel; ++l) t += sa[r][l] * sw[l][m];
    }
    st[r][m] = m < b ? t : 0.0;
  }
  __syncthreads();
#pragma unroll 4
  for (int m = 0; m < kGJPanel; ++m) {
    double t[4], p[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) t[r] = st[ty + 16 * r][m];
#pragma unroll
    for (int c = 0; c < 4; ++c) p[c] = sb[m][tx + 16 * c];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) v[r][c] -= t[r] * p[c];
  }
  const int k1 = k0 + kGJPanel;   // next pivot block; 32 divides 64, so it lies in one tile
  const int bn = min(kGJPanel, n - k1);
  const bool next = bn > 0 && i0 == k1 / kGJTile * kGJTile && j0 == i0;
  const int off = k1 - i0;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = i0 + ty + 16 * r, j = j0 + tx + 16 * c;
      if (j >= k0 && j < k0 + b) v[r][c] = -st[ty + 16 * r][j - k0];
      if (i < n && j < n) B[(size_t)i * n + j] = v[r][c];
      if (next) {
        const int pr = ty + 16 * r - off, pc = tx + 16 * c - off;
        if (pr >= 0 && pr < kGJPanel && pc >= 0 && pc < kGJPanel)
          sp[0][pr][pc] = (pr < bn && pc < bn) ? v[r][c] : (pr == pc ? 1.0 : 0.0);
      }
    }
  if (!next) return;   // the same for the whole CTA
  __syncthreads();
  // Gauss-Jordan on the 32x32 block, ping-pong between two copies
  for (int k = 0; k < kGJPanel; ++k) {
    const double(*o)[kGJPanel + 1] = sp[k & 1];
    double(*w)[kGJPanel + 1] = sp[(k & 1) ^ 1];
    const double ip = 1.0 / o[k][k];
#pragma unroll
    for (int q = threadIdx.x; q < kGJPanel * kGJPanel; q += 256) {
      const int r = q / kGJPanel, c = q % kGJPanel;
      double x;
      if (r == k) x = (c == k) ? ip : o[k][c] * ip;
      else if (c == k) x = -o[r][k] * ip;
      else x = o[r][c] - o[r][k] * o[k][c] * ip;
      w[r][c] = x;
    }
    __syncthreads();
  }
  for (int q = threadIdx.x; q < kGJPanel * kGJPanel; q += 256) Wn[q] = sp[0][q / kGJPanel][q % kGJPanel];
}

// out = (A + A^T) / 2: the inverse of the SPD coarse matrix is symmetric in exact
// arithmetic; the elimination's rounding is not, and a symmetric coarse solve
// keeps the V-cycle a symmetric preconditioner.  32x32 tiles through shared memory.
__global__ void __launch_bounds__(256) k_symmetrize(const double* A, double* out, int n) {
  grid_dep_wait();
  __shared__ double s[32][33];
  const int i0 = blockIdx.y * 32, j0 = blockIdx.x * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int r = ty; r < 32; r += 8)
    if (j0 + r < n && i0 + tx < n) s[r][tx] = A[(size_t)(j0 + r) * n + i0 + tx];
  __syncthreads();
#pragma unroll
  for (int r = ty; r < 32; r += 8)
    if (i0 + r < n && j0 + tx < n)
      out[(size_t)(i0 + r) * n + j0 + tx] = 0.5 * (A[(size_t)(i0 + r) * n + j0 + tx] + s[tx][r]);
}

// x = Inv b, one CTA per row: each thread reads a few entries of the row (all
// loads in flight at once), then a block reduction.
template <typename T>
__global__ void __launch_bounds__(128) k_dense_apply(const double* __restrict__ Inv, const T* b,
                                                     T* x, int n) {
  grid_dep_launch();
  const int row = blockIdx.x;
  const double* a = Inv + (size_t)row * n;
  // the row is constant during a solve: its first 12 x 128 entries (all of it
  // up to the default coarse_max) are fetched before the wait
  constexpr int kPre = 12;
  double av[kPre];
#pragma unroll
  for (int k = 0; k < kPre; ++k) {
    const int j = threadIdx.x + 128 * k;
    av[k] = j < n ? ld_stream(a + j) : 0.0;
  }
  grid_dep_sync();
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < kPre; ++k) {
    const int j = threadIdx.x + 128 * k;
    if (j < n) s += av[k] * (double)b[j];
  }
  for (int j = threadIdx.x + 128 * kPre; j < n; j += 128) s += a[j] * (double)b[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  __shared__ double part[4];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) x[row] = (T)(part[0] + part[1] + part[2] + part[3]);
}

// ---- host side ---------------------------------------------------------------
static int tpb(int64_t n) { return (int)div_up(n, 256); }

template <typename T>
static T* level_K(MGLevel& L);
template <>
double* level_K<double>(MGLevel& L) { return L.K64; }
template <>
float* level_K<float>(MGLevel& L) { return L.K32; }
template <typename T>
static T* level_dinv(MGLevel& L);
template <>
double* level_dinv<double>(MGLevel& L) { return L.dinv64; }
template <>
float* level_dinv<float>(MGLevel& L) { return L.dinv32; }

void mg_free(Ctx& c) {
  ++c.alloc_gen;
  for (size_t l = 0; l < c.mg.size(); ++l) {
    MGLevel& L = c.mg[l];
    if (l > 0) { cudaFree(L.K64); cudaFree(L.K32); }
    cudaFree(L.dinv64); cudaFree(L.dinv32); cudaFree(L.cheb);
    cudaFree(L.x); cudaFree(L.b); cudaFree(L.r); cudaFree(L.d); cudaFree(L.t); cudaFree(L.S);
  }
  c.mg.clear();
  cudaFree(c.coarse_inv);
  c.coarse_inv = nullptr;
  c.coarse_n = 0;
  c.mg_prec = -1;
}

// ---- smoother bounds -----------------------------------------------------------
// lambda_max(D^-1 A) from kLanSteps steps of Jacobi-PCG on a pseudo-random start
// vector: the Lanczos coefficients stay on the device, in the level's table,
// and one kernel turns those of all levels into Chebyshev coefficients, so the
// set-up enqueues without waiting for the GPU.
constexpr int kLanSteps = 10;
enum LanSlot { LAN_RZ = 0, LAN_PAP = 1, LAN_M = 2, LAN_STOP = 3, LAN_ALPHA = 4, LAN_BETA = LAN_ALPHA + kLanSteps,
               LAN_COUNT = LAN_BETA + kLanSteps };
constexpr int kChebCoefs = 2 * (kMaxCheb + 1);   // of a level's table: the coefficients, then the LAN_ slots

// r = deterministic pseudo-random vector (zero on fixed DOFs), p = z = D^-1 r, Ap = 0, r.z
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_lan_start(const T* __restrict__ dinv, T* r, T* p, T* Ap, int64_t nnod,
                                                           int A, int pin, double* lan, double* partial,
                                                           unsigned int* counter) {
  typedef typename V2<T>::T X2;
  double v[1] = {0.0};
  for (int64_t n = blockIdx.x * (int64_t)kRedThreads + threadIdx.x; n < nnod; n += (int64_t)gridDim.x * kRedThreads) {
    const int a = (int)(n % A), b = (int)(n / A);
    X2 rv, zv;
    T u[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint64_t z = (uint64_t)(2 * n + c) * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
      z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
      z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
      z ^= z >> 31;
      u[c] = dof_fixed(a, b, c, A - 1, pin) ? (T)0 : (T)((double)(z >> 11) * (1.0 / 9007199254740992.0) - 0.5);
    }
    double z0, z1;
    bj_apply<T>(dinv, n, (double)u[0], (double)u[1], z0, z1);
    rv.x = u[0]; rv.y = u[1];
    zv.x = (T)z0; zv.y = (T)z1;
    reinterpret_cast<X2*>(r)[n] = rv;
    reinterpret_cast<X2*>(p)[n] = zv;
    zv.x = zv.y = (T)0;
    reinterpret_cast<X2*>(Ap)[n] = zv;
    v[0] += (double)u[0] * (double)(T)z0 + (double)u[1] * (double)(T)z1;
  }
  double* o[1] = {lan + LAN_RZ};
  if (grid_finish<1>(v, partial, counter, o) && threadIdx.x == 0) {
    lan[LAN_M] = 0.0;
    lan[LAN_STOP] = lan[LAN_RZ] > 0.0 ? 0.0 : 1.0;
  }
}

// p.Ap; stops the recurrence where it is not positive
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_lan_pap(const T* p, const T* Ap, int64_t n, double* lan,
                                                         double* partial, unsigned int* counter) {
  if (lan[LAN_STOP] != 0.0) return;
  double v[1] = {0.0};
  for (int64_t i = blockIdx.x * (int64_t)kRedThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kRedThreads)
    v[0] += (double)p[i] * (double)Ap[i];
  double* o[1] = {lan + LAN_PAP};
  if (grid_finish<1>(v, partial, counter, o) && threadIdx.x == 0 && !(lan[LAN_PAP] > 0.0)) lan[LAN_STOP] = 1.0;
}

// r -= alpha Ap; z = D^-1 r; r.z; the last block records alpha and beta
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_lan_update(T* r, const T* Ap, const T* __restrict__ dinv, T* z,
                                                            int64_t nnod, double* lan, double* partial,
                                                            unsigned int* counter) {
  if (lan[LAN_STOP] != 0.0) return;
  typedef typename V2<T>::T X2;
  const double rz = lan[LAN_RZ], alpha = rz / lan[LAN_PAP];
  double v[1] = {0.0};
  for (int64_t n = blockIdx.x * (int64_t)kRedThreads + threadIdx.x; n < nnod; n += (int64_t)gridDim.x * kRedThreads) {
    X2 rv = reinterpret_cast<X2*>(r)[n];
    const X2 av = reinterpret_cast<const X2*>(Ap)[n];
    const double r0 = (double)rv.x - alpha * (double)av.x, r1 = (double)rv.y - alpha * (double)av.y;
    double z0, z1;
    bj_apply<T>(dinv, n, r0, r1, z0, z1);
    rv.x = (T)r0; rv.y = (T)r1;
    reinterpret_cast<X2*>(r)[n] = rv;
    X2 zv;
    zv.x = (T)z0; zv.y = (T)z1;
    reinterpret_cast<X2*>(z)[n] = zv;
    v[0] += (double)rv.x * (double)zv.x + (double)rv.y * (double)zv.y;
  }
  // every block has read rz before the ticket of the last one is drawn, so the
  // result may replace it
  double* o[1] = {lan + LAN_RZ};
  if (grid_finish<1>(v, partial, counter, o) && threadIdx.x == 0) {
    const int m = (int)lan[LAN_M];
    lan[LAN_ALPHA + m] = alpha;
    lan[LAN_BETA + m] = lan[LAN_RZ] / rz;
    lan[LAN_M] = (double)(m + 1);
    if (!(lan[LAN_RZ] > 0.0)) lan[LAN_STOP] = 1.0;
  }
}

// p = z + beta p, Ap = 0
template <typename T>
__global__ void k_lan_dir(const T* z, T* p, T* Ap, int64_t n, const double* lan) {
  if (lan[LAN_STOP] != 0.0) return;
  const double beta = lan[LAN_BETA + (int)lan[LAN_M] - 1];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) {
    p[i] = z[i] + (T)(beta * (double)p[i]);
    Ap[i] = (T)0;
  }
}

template <typename T>
static void estimate_lmax(Ctx& c, MGLevel& L) {
  const int64_t nn = L.g.nnod, n = 2 * nn;
  T* r = (T*)L.r; T* p = (T*)L.d; T* z = (T*)L.b; T* Ap = (T*)L.t;
  const T* dinv = level_dinv<T>(L);
  double* lan = L.cheb + kChebCoefs;
  klaunch(k_lan_start<T>, red_grid(n), kRedThreads, 0, c.stream, dinv, r, p, Ap, nn, (int)L.g.A(), L.g.pin, lan,
          c.partial, c.counter);
  for (int k = 0; k < kLanSteps; ++k) {
    launch_apply_K_acc<T, T>(L.g, level_K<T>(L), p, Ap, c.stream);
    klaunch(k_lan_pap<T>, red_grid(n), kRedThreads, 0, c.stream, p, Ap, n, lan, c.partial, c.counter);
    klaunch(k_lan_update<T>, red_grid(n), kRedThreads, 0, c.stream, r, Ap, dinv, z, nn, lan, c.partial, c.counter);
    if (k + 1 < kLanSteps) klaunch(k_lan_dir<T>, tpb(n), 256, 0, c.stream, z, p, Ap, n, lan);
  }
  DP_LAUNCH_CHECK();
}

// Chebyshev recurrence coefficients on [lo, hi] * lambda_max (three-term form),
// one warp per level.  lambda_max of the Lanczos tridiagonal matrix by Sturm
// counts: 32 trial values a round, 12 rounds (33^-12 of the Gershgorin interval).
struct ChebArgs {
  double* cheb[16];
  int degree[16];
};
__global__ void __launch_bounds__(32) k_cheb_coefs(ChebArgs args, double frac_lo, double frac_hi) {
  double* coef = args.cheb[blockIdx.x];
  const double* lan = coef + kChebCoefs;
  const int lane = threadIdx.x, m = (int)lan[LAN_M], degree = args.degree[blockIdx.x];
  double lmax = 2.0;
  if (m > 0) {
    double a[kLanSteps], b2[kLanSteps], lo = 0.0, hi = 0.0, left = 0.0;
    for (int j = 0; j < m; ++j) {
      a[j] = 1.0 / lan[LAN_ALPHA + j] + (j > 0 ? lan[LAN_BETA + j - 1] / lan[LAN_ALPHA + j - 1] : 0.0);
      const double b = j < m - 1 ? sqrt(lan[LAN_BETA + j]) / lan[LAN_ALPHA + j] : 0.0;
      b2[j] = b * b;
      hi = fmax(hi, a[j] + left + b);
      lo = fmin(lo, a[j] - left - b);
      left = b;
    }
    for (int round = 0; round < 12; ++round) {
      const double x = lo + (hi - lo) * ((lane + 1) * (1.0 / 33.0));
      int cnt = 0;
      double d = 1.0;
      for (int j = 0; j < m; ++j) {
        d = a[j] - x - (j > 0 ? b2[j - 1] / d : 0.0);
        if (d == 0.0) d = 1e-300;
        if (d < 0) ++cnt;
      }
      const unsigned above = __ballot_sync(0xffffffffu, cnt >= m);   // trial values >= lambda_max
      const int first = above ? __ffs(above) - 1 : 32;
      const double xl = __shfl_sync(0xffffffffu, x, first > 0 ? first - 1 : 0);
      const double xh = __shfl_sync(0xffffffffu, x, first < 32 ? first : 31);
      if (first > 0) lo = xl;
      if (first < 32) hi = xh;
    }
    lmax = hi;
  }
  if (lane != 0) return;
  const double lmx = frac_hi * lmax, lmn = frac_lo * lmax;
  const double theta = 0.5 * (lmx + lmn), delta = 0.5 * (lmx - lmn), sigma = theta / delta;
  double rho_prev = 1.0 / sigma;
  coef[0] = 1.0 / theta;
  for (int k = 1; k < degree; ++k) {
    const double rho = 1.0 / (2.0 * sigma - rho_prev);
    coef[2 * k] = rho * rho_prev;
    coef[2 * k + 1] = 2.0 * rho / delta;
    rho_prev = rho;
  }
}

template <typename T>
static void setup_level_vectors(MGLevel& L) {
  const size_t bytes = sizeof(T) * 2 * L.g.nnod;
  DP_CUDA(cudaMalloc(&L.x, bytes));
  DP_CUDA(cudaMalloc(&L.b, bytes));
  DP_CUDA(cudaMalloc(&L.r, bytes));
  DP_CUDA(cudaMalloc(&L.d, bytes));
  DP_CUDA(cudaMalloc(&L.t, bytes));
}

template <typename T>
static void mg_setup_t(Ctx& c, const MGOptions& o) {
  const int prec = std::is_same<T, float>::value ? 1 : 0;
  // level geometry (reuse if unchanged)
  if (c.mg.empty() || c.mg_prec != prec || c.mg_coarse_max != o.coarse_max) {
    mg_free(c);
    MGLevel L0;
    L0.g = c.fine;
    c.mg.push_back(L0);
    while (true) {
      const Level& g = c.mg.back().g;
      if (g.ncr % 2 || g.nct % 2 || g.nct / 2 < 4) break;
      if ((int)c.mg.size() >= o.max_levels) break;
      Level h;
      h.ncr = g.ncr / 2;
      h.nct = g.nct / 2;
      h.nel = 2 * (int64_t)h.ncr * h.nct;
      h.nnod = h.A() * h.B();
      h.pin = g.pin;
      if (2 * g.nnod <= o.coarse_max) break;
      MGLevel Lh;
      Lh.g = h;
      c.mg.push_back(Lh);
    }
    for (size_t l = 0; l < c.mg.size(); ++l) {
      MGLevel& L = c.mg[l];
      if (l > 0) {
        DP_CUDA(cudaMalloc(prec ? (void**)&L.K32 : (void**)&L.K64, sizeof(T) * kstore<T>(L.g.nel)));
      }
      DP_CUDA(cudaMalloc(prec ? (void**)&L.dinv32 : (void**)&L.dinv64, sizeof(T) * 3 * L.g.nnod));
      DP_CUDA(cudaMalloc(&L.cheb, sizeof(double) * (kChebCoefs + LAN_COUNT)));
      DP_CUDA(cudaMemsetAsync(L.cheb, 0, sizeof(double) * (kChebCoefs + LAN_COUNT), c.stream));
      setup_level_vectors<T>(L);
      if (l + 1 < c.mg.size() && L.g.nnod <= kStencilMaxNodes)
        DP_CUDA(cudaMalloc(&L.S, sizeof(T) * stencil_store<T>(L.g.ncr, L.g.nct)));
    }
    c.coarse_n = 2 * c.mg.back().g.nnod;
    if (c.coarse_n <= o.coarse_max) {
      DP_CUDA(cudaMalloc(&c.coarse_inv, sizeof(double) * (c.coarse_n * c.coarse_n * 2 + 2 * kGJPanel * kGJPanel)));
    } else {
      c.coarse_n = 0;
    }
    DP_CUDA(cudaFuncSetAttribute(k_galerkin<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)GalerkinTile<T>::kSmem));
    DP_CUDA(cudaFuncSetAttribute(k_gj_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGJSmem));
    c.mg_prec = prec;
    c.mg_coarse_max = o.coarse_max;
  }
  // fine operator pointer, apply tiles
  if (prec) c.mg[0].K32 = c.K32; else c.mg[0].K64 = c.K64;
  for (MGLevel& L : c.mg) {
    L.g.warps = o.apply_warps;
    L.g.warps_t = o.apply_warps_t;
    L.g.det = c.fine.det;   // one scratch (sized for the fine level) serves every level in turn
    L.g.mfD64 = L.g.mfT64 = nullptr;
    L.g.mfD32 = L.g.mfT32 = nullptr;
    L.g.red64 = nullptr;
    L.g.red32 = nullptr;
  }
  // the fine level applies matrix-free when the fine context level does
  c.mg[0].g.mfD64 = c.fine.mfD64;
  c.mg[0].g.mfT64 = c.fine.mfT64;
  c.mg[0].g.red64 = c.fine.red64;
  c.mg[0].g.red32 = c.fine.red32;
  c.mg[0].g.mfD32 = c.fine.mfD32;
  c.mg[0].g.mfT32 = c.fine.mfT32;
  // Galerkin coarse operators
  for (size_t l = 1; l < c.mg.size(); ++l) {
    MGLevel& Lf = c.mg[l - 1];
    MGLevel& Lc = c.mg[l];
    klaunch(k_galerkin<T>, (int)div_up((int64_t)Lc.g.ncr * Lc.g.nct, 32), kGalThreads, GalerkinTile<T>::kSmem,
            c.stream, level_K<T>(Lf), level_K<T>(Lc), Lc.g.ncr, Lc.g.nct, Lf.g.ncr, Lc.g.pin);
    DP_LAUNCH_CHECK();
  }
  for (MGLevel& L : c.mg)
    if (L.S) launch_stencil_assemble<T>(L.g, level_K<T>(L), (T*)L.S, c.stream);
  // nodal diagonal blocks, eigenvalue estimates and Chebyshev coefficients
  const int deg = std::max(1, std::min(o.cheb_degree, kMaxCheb));
  const int deg_coarse = o.cheb_degree_coarse > 0 ? std::max(1, std::min(o.cheb_degree_coarse, kMaxCheb)) : deg;
  ChebArgs ca{};
  int nsmooth = 0;
  for (size_t l = 0; l < c.mg.size(); ++l) {
    MGLevel& L = c.mg[l];
    L.degree = l == 0 ? deg : deg_coarse;
    klaunch(k_diag_invert<T>, tpb((int64_t)(L.g.ncr + 1) * L.g.nct), 256, 0, c.stream, level_K<T>(L),
            level_dinv<T>(L), L.g.ncr, L.g.nct, L.g.pin, o.block_jacobi);
    DP_LAUNCH_CHECK();
    if (l + 1 == c.mg.size() && c.coarse_n > 0) continue;   // solved directly, never smoothed
    estimate_lmax<T>(c, L);
    ca.cheb[nsmooth] = L.cheb;
    ca.degree[nsmooth++] = L.degree;
  }
  if (nsmooth > 0) klaunch(k_cheb_coefs, nsmooth, 32, 0, c.stream, ca, o.cheb_lo, o.cheb_hi);
  DP_LAUNCH_CHECK();
  c.mg_degree = deg + 16 * deg_coarse;  // both degrees shape the captured graph
  // coarse dense inverse
  if (c.coarse_n > 0) {
    MGLevel& L = c.mg.back();
    const int n = (int)c.coarse_n, npanel = (int)div_up(n, kGJPanel);
    double* D = c.coarse_inv;
    double* Inv = D + (size_t)n * n;
    double* W = Inv + (size_t)n * n;   // two panel inverses, in turn
    // ping-pong between D and Inv such that the last panel writes D
    double* cur = (npanel & 1) ? Inv : D;
    double* oth = (npanel & 1) ? D : Inv;
    DP_CUDA(cudaMemsetAsync(cur, 0, sizeof(double) * n * n, c.stream));
    klaunch(k_dense_assemble<T>, dim3((unsigned)div_up(st_nodes(0, L.g.ncr, L.g.nct), 64), 4), 64, 0, c.stream,
            level_K<T>(L), cur, L.g.ncr, L.g.nct);
    klaunch(k_dense_fix_diag, (int)div_up(n, 256), 256, 0, c.stream, cur, n);
    klaunch(k_gj_panel_inverse, 1, dim3(kGJPanel, kGJPanel), 0, c.stream, cur, W, n, 0, std::min(kGJPanel, n));
    const unsigned tiles = (unsigned)div_up(n, kGJTile);
    for (int p = 0; p < npanel; ++p) {
      klaunch(k_gj_panel, dim3(tiles, tiles), 256, kGJSmem, c.stream, cur, oth,
              W + (p & 1) * kGJPanel * kGJPanel, W + ((p & 1) ^ 1) * kGJPanel * kGJPanel, n, p * kGJPanel);
      std::swap(cur, oth);
    }
    const unsigned blk = (unsigned)div_up(n, 32);
    klaunch(k_symmetrize, dim3(blk, blk), 256, 0, c.stream, D, Inv, n);
    DP_LAUNCH_CHECK();
  }
}

void mg_setup(Ctx& c, int precision, const MGOptions& o) {
  if (precision == 1) mg_setup_t<float>(c, o);
  else mg_setup_t<double>(c, o);
}

// Levels whose smoother runs on node stencils: those that have them, except
// with one Chebyshev step (the deferred x update below needs a second one) and
// with a matrix-free fine level.
static bool stencil_level(const Ctx& c, const MGLevel& L) {
  return L.S && L.degree >= 2 && !(&L == &c.mg[0] && (L.g.mfD64 || L.g.mfD32));
}

// Chebyshev smoothing on node stencils (same recurrence and modes as
// chebyshev(), r read from b in mode 2).  d alternates between L.d and L.t: a
// step gathers the old d from neighbours that other threads are replacing.  In
// mode 2 the first step gathers x, so x gains d_1 together with d_2.
// Pre-smoothing (modes 0, 1) ends with r = b - A x, the true residual.
template <typename T>
static bool chebyshev_stencil(Ctx& c, MGLevel& L, const T* b, T* x, int mode, const RzOut* rz = nullptr) {
  T* r = (T*)L.r;
  T* d = (T*)L.d;
  T* dn = (T*)L.t;
  const T* S = (const T*)L.S;
  const T* dinv = level_dinv<T>(L);
  const T* none = nullptr;
  if (mode == 0) klaunch(k_cheb_first<T>, tpb(L.g.nnod), 256, 0, c.stream, b, dinv, x, r, d, L.cheb, L.g.nnod);
  if (mode == 2) launch_stencil_step<ST_FIRST_X, T>(L.g, S, x, b, r, (T*)nullptr, d, dinv, L.cheb, c.stream);
  bool summed = false;
  for (int k = 1; k < L.degree; ++k) {
    const double* coef = L.cheb + 2 * k;
    if (mode == 2 && k == 1) {
      launch_stencil_step<ST_STEP_X, T>(L.g, S, d, none, r, x, dn, dinv, coef, c.stream);
    } else if (rz && k + 1 == L.degree) {
      launch_stencil_step<ST_STEP_RZ, T>(L.g, S, d, none, r, x, dn, dinv, coef, c.stream, *rz);
      summed = true;
    } else {
      launch_stencil_step<ST_STEP, T>(L.g, S, d, none, r, x, dn, dinv, coef, c.stream);
    }
    std::swap(d, dn);
  }
  if (mode != 2)
    launch_stencil_step<ST_RESIDUAL, T>(L.g, S, d, none, r, (T*)nullptr, (T*)nullptr, dinv, L.cheb, c.stream);
  DP_LAUNCH_CHECK();
  return summed;
}

// Levels whose x is put together late (see the vector steps above); not the
// coarsest, which has no prolongation to complete it.
static bool late_x(const Ctx& c, const MGLevel& L) {
  return !stencil_level(c, L) && (L.degree == 2 || L.degree == 3) && &L != &c.mg.back();
}

// Chebyshev smoothing of A x = b on level L.  mode 0: start from x = 0;
// mode 1: start from x = 0 with the first step already taken (fused into the
// restriction that produced b); mode 2: start from the given x, with L.r
// holding b on entry (the prolongation copies it there).  The recurrence
// coefficients live in L.cheb on the device, so this sequence is the same for
// every assembly and is captured once into the solve graph.
// On exit of modes 0 and 1 r = b - A (x - d_last), i.e. the true residual is
// r - A d_last; returns d_last, which for late_x levels lies in x (x itself is
// then L.d (+ L.t) + x, completed by the prolongation).
template <typename T>
static const T* chebyshev(Ctx& c, MGLevel& L, const T* b, T* x, int mode) {
  if (stencil_level(c, L)) {
    chebyshev_stencil<T>(c, L, b, x, mode);
    return nullptr;
  }
  const int64_t nn = L.g.nnod;
  T* r = (T*)L.r;
  T* d = (T*)L.d;
  const T* dinv = level_dinv<T>(L);
  const bool late = late_x(c, L);
  const T* none = nullptr;
  if (mode == 0) {
    klaunch(k_cheb_first<T>, tpb(nn), 256, 0, c.stream, b, dinv, late ? (T*)nullptr : x, r, d, L.cheb, nn);
  } else if (mode == 2) {
    launch_apply_K_sub<T, T>(L.g, level_K<T>(L), x, r, c.stream);
    klaunch(k_cheb_first_x<T>, tpb(nn), 256, 0, c.stream, (const T*)r, dinv, late ? (T*)nullptr : x, d, L.cheb, nn);
  }
  const T* before = nullptr;   // the step before d (late form)
  for (int k = 1; k < L.degree; ++k) {
    launch_apply_K_sub<T, T>(L.g, level_K<T>(L), (const T*)d, r, c.stream);
    const double* coef = L.cheb + 2 * k;
    if (!late) {
      klaunch(k_cheb_step<CH_IN_PLACE, T>, tpb(nn), 256, 0, c.stream, (const T*)r, dinv, x, d, (T*)nullptr, none, coef,
              nn);
    } else if (mode == 2 && k + 1 == L.degree) {
      klaunch(k_cheb_step<CH_LAST, T>, tpb(nn), 256, 0, c.stream, (const T*)r, dinv, x, d, (T*)nullptr, before, coef,
              nn);
    } else {
      T* dn = k + 1 == L.degree ? x : (T*)L.t;
      klaunch(k_cheb_step<CH_NEXT, T>, tpb(nn), 256, 0, c.stream, (const T*)r, dinv, (T*)nullptr, d, dn, none, coef,
              nn);
      before = d;
      d = dn;
    }
  }
  DP_LAUNCH_CHECK();
  return d;
}

// Levels smoothed by whole passes (halo.cu): stencils, the default degree, small enough.
template <typename T>
static bool halo_level(const Ctx& c, size_t l, const MGOptions& o) {
  const MGLevel& L = c.mg[l];
  return l + 1 < c.mg.size() && l < tail_start(c, o) && stencil_level(c, L) && L.degree == kHaloDegree &&
         halo_fits<T>(L.g);
}

// first_done: the level's first pre-smoothing step was fused into the restriction.
// rz (fine level): see mg.cuh; returns whether the last kernel took it.
template <typename T>
static bool vcycle(Ctx& c, size_t l, const T* b, T* x, const MGOptions& o, bool first_done,
                   const RzOut* rz = nullptr) {
  if (l == tail_start(c, o)) {
    launch_vcycle_tail<T>(c, l, b, x, first_done, o);
    return false;
  }
  MGLevel& L = c.mg[l];
  if (L.g.det) rz = nullptr;   // an atomic per block: the sum would depend on scheduling
  const bool dense_coarsest = c.coarse_n > 0;
  if (l + 1 == c.mg.size()) {
    if (dense_coarsest) {
      // dense inverse: identity rows on constrained DOFs keep them at zero
      const int nn = (int)c.coarse_n;
      const double* Inv = c.coarse_inv + (size_t)nn * nn;
      klaunch(k_dense_apply<T>, nn, 128, 0, c.stream, Inv, b, x, nn);
      DP_LAUNCH_CHECK();
    } else {
      chebyshev<T>(c, L, b, x, first_done ? 1 : 0);
      for (int s = 1; s < o.coarse_sweeps; ++s) {
        DP_CUDA(cudaMemcpyAsync(L.r, b, sizeof(T) * 2 * L.g.nnod, cudaMemcpyDeviceToDevice, c.stream));
        chebyshev<T>(c, L, b, x, 2);
      }
    }
    return false;
  }
  MGLevel& C = c.mg[l + 1];
  T* r = (T*)L.r;
  T* bc = (T*)C.b;
  T* xc = (T*)C.x;
  // pre-smoothing, r -= A d_last (the true residual), then restrict it (and take
  // the coarse level's first smoothing step in the same pass unless it is
  // solved densely or smoothed by whole passes)
  const bool st = stencil_level(c, L);   // its pre-smoothing leaves the true residual in r
  const bool halo = halo_level<T>(c, l, o);
  const unsigned halo_threads = 32 * halo_warps(L.g.ncr);
  if (halo) {   // the smoothed x goes to L.d
    klaunch(k_halo_down<T>, (unsigned)L.g.nct, halo_threads, 0, c.stream, (const T*)L.S, b, r, (T*)L.d,
            level_dinv<T>(L), (const double*)L.cheb, L.g.ncr, L.g.nct);
  } else {
    const T* d_last = chebyshev<T>(c, L, b, x, first_done ? 1 : 0);
    if (!st) launch_apply_K_sub<T, T>(L.g, level_K<T>(L), d_last, r, c.stream);
  }
  const bool fuse = !(l + 2 == c.mg.size() && dense_coarsest) && !halo_level<T>(c, l + 1, o);
  // the cluster tail's smoother accumulates A d into t, which starts at zero
  T* tc = (l + 1 == tail_start(c, o)) ? (T*)C.t : nullptr;
  const int nA0 = (int)((C.g.A() + 1) >> 1);  // coarse nodes per parity class (upper bound)
  // a coarse level that puts its x together late does not read it before the prolongation from below
  T* xc1 = late_x(c, C) && l + 1 != tail_start(c, o) ? nullptr : xc;
  // the tiled form needs whole tiles along theta (its patch then wraps at most once)
  const bool small = C.g.nnod < 32768 || C.g.B() % kRTile != 0;
  if (small) {
    dim3 grid((unsigned)div_up(4 * (int64_t)nA0 * (C.g.B() >> 1), 256), 4);
    klaunch(k_restrict_g<T>, grid, 256, 0, c.stream, (const T*)r, bc, (int)L.g.A(),
            (int)L.g.B(), (int)C.g.A(), (int)C.g.B(), C.g.pin, fuse ? 1 : 0, (const T*)level_dinv<T>(C), xc1, (T*)C.r,
            (T*)C.d, tc, (const double*)C.cheb);
  } else {
    dim3 grid((unsigned)div_up(C.g.A(), kRTile), (unsigned)div_up(C.g.B(), kRTile));
    klaunch(k_restrict_tile<T>, grid, 256, 0, c.stream, (const T*)r, bc, (int)L.g.A(),
            (int)L.g.B(), (int)C.g.A(), (int)C.g.B(), C.g.pin, fuse ? 1 : 0, (const T*)level_dinv<T>(C), xc1,
            (T*)C.r, (T*)C.d, tc, (const double*)C.cheb);
  }
  DP_LAUNCH_CHECK();
  vcycle<T>(c, l + 1, bc, xc, o, fuse);
  if (halo) {
    klaunch(k_halo_up<T>, (unsigned)L.g.nct, halo_threads, 0, c.stream, (const T*)L.S, b, (const T*)xc, (const T*)L.d,
            x, level_dinv<T>(L), (const double*)L.cheb, L.g.ncr, L.g.nct, C.g.ncr, (int)C.g.A(), (int)C.g.B(),
            L.g.pin, rz ? *rz : RzOut());
    DP_LAUNCH_CHECK();
    return rz != nullptr;
  }
  klaunch(k_prolong_add<T>, tpb(L.g.nnod), 256, 0, c.stream, (const T*)xc, x,
          late_x(c, L) ? (const T*)L.d : (const T*)nullptr,
          late_x(c, L) && L.degree == 3 ? (const T*)L.t : (const T*)nullptr, b, st ? (T*)nullptr : r, (int)L.g.A(),
          (int)L.g.B(), C.g.ncr, (int)C.g.A(), (int)C.g.B(), L.g.pin);
  DP_LAUNCH_CHECK();
  if (!st) rz = nullptr;
  return st ? chebyshev_stencil<T>(c, L, b, x, 2, rz) : (chebyshev<T>(c, L, b, x, 2), false);
}

bool mg_apply(Ctx& c, const double* b, double* x, const MGOptions& o, bool first_done, const RzOut* rz) {
  return vcycle<double>(c, 0, b, x, o, first_done, rz);
}
bool mg_apply_f(Ctx& c, const float* b, float* x, const MGOptions& o, bool first_done, const RzOut* rz) {
  return vcycle<float>(c, 0, b, x, o, first_done, rz);
}

template <typename T>
FirstStep<T> mg_first_step(Ctx& c, T* x, const MGOptions& o) {
  FirstStep<T> f;
  if (c.mg.size() < 2 || tail_start(c, o) == 0 || !stencil_level(c, c.mg[0]) || halo_level<T>(c, 0, o)) return f;
  MGLevel& L = c.mg[0];
  f.dinv = level_dinv<T>(L);
  f.r = (T*)L.r;
  f.d = (T*)L.d;
  f.x = x;
  f.coef = L.cheb;
  return f;
}
template FirstStep<float> mg_first_step<float>(Ctx&, float*, const MGOptions&);
template FirstStep<double> mg_first_step<double>(Ctx&, double*, const MGOptions&);
template <typename T>
void launch_first_step(Ctx& c, const T* b, const FirstStep<T>& f) {
  const int64_t nn = c.fine.nnod;
  klaunch(k_cheb_first<T>, tpb(nn), 256, 0, c.stream, b, f.dinv, f.x, f.r, f.d, f.coef, nn);
}
template void launch_first_step<float>(Ctx&, const float*, const FirstStep<float>&);
template void launch_first_step<double>(Ctx&, const double*, const FirstStep<double>&);

}  // namespace dp
