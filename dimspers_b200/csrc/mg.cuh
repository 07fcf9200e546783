// Multigrid hierarchy interface and lattice helpers shared by its kernels.
#pragma once
#include "ctx.cuh"

namespace dp {

constexpr int kMaxCheb = 8;
// Largest level (lattice nodes) whose smoother runs on node stencils: the
// 32x256 level (33,280 nodes) and below.  Per inner iteration of the whole
// solve when they came in: 16x128 FP64 80.7 -> 67.5 us, 32x256 103 -> 92.8 us.
// On larger fine levels the bytes (184 a node against 112 of the reduced element
// matrices) weigh more than the launches; fast path, element form -> stencils on the fine level too:
// 42k nodes (36x288) 89.5 -> 84.7 us, 52k (40x320) 100.2 -> 97.7, 74k (48x384)
// 93.8 -> 89.0, 101k (56x448) 115.0 -> 114.3, 132k (64x512) 112.7 -> 116.4.
// The two meet near 100k nodes; the line is below that, at the largest level of
// the meshes that halve down from the benchmark's.
constexpr int64_t kStencilMaxNodes = 40000;

struct MGOptions {
  int cheb_degree = 3;      // Chebyshev steps per smoothing (each one A-apply)
  int cheb_degree_coarse = 0;  // on the levels below the finest (0: cheb_degree)
  double cheb_lo = 0.15;    // smoothing interval [lo, hi] * lambda_max(D^-1 A)
  double cheb_hi = 1.1;
  int block_jacobi = 1;     // 1: 2x2 nodal blocks (u_theta, u_r); 0: point Jacobi
  int max_levels = 16;
  int64_t coarse_max = 1536;// largest dense coarsest system
  int coarse_sweeps = 4;    // smoothing sweeps when the coarsest is not dense
  int64_t tail_max_el = 0;  // levels up to this many elements run as one cluster kernel (0: off)
  int apply_warps = 4;      // tile of the element-by-element applies (Level::warps)
  int apply_warps_t = 1;    // (Level::warps_t)
};

// Local node offsets (radial, angular) inside the cell for triangle type t.
__host__ __device__ inline int kLocA_dev(int t, int k) {
  const int A0[6] = {0, 0, 2, 0, 1, 1}, A1[6] = {0, 2, 2, 1, 2, 1};
  return t == 0 ? A0[k] : A1[k];
}
__host__ __device__ inline int kLocB_dev(int t, int k) {
  const int B0[6] = {0, 2, 0, 1, 1, 0}, B1[6] = {2, 2, 0, 2, 1, 1};
  return t == 0 ? B0[k] : B1[k];
}
__host__ __device__ inline void element_nodes_mg(int e, int ncr, int A, int B, int nd[6]) {
  const int q = e >> 1, t = e & 1;
  const int ir = q % ncr, it = q / ncr;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    int b = 2 * it + kLocB_dev(t, k);
    if (b >= B) b -= B;
    nd[k] = 2 * ir + kLocA_dev(t, k) + A * b;
  }
}

void upload_mg_constants();
void mg_setup(Ctx& c, int precision, const MGOptions& o);
void mg_free(Ctx& c);
// first_done: the caller has taken the fine level's first smoother step (mg_first_step).
// rz given: the cycle's last kernel also adds r . s x to *rz->out (s = sqrt(*rz->yy), 1 without
// yy; r in FP64) if it is of a kind that can (the passes and steps on stencils, whose few blocks
// make few atomics; on larger levels the launch saved is below 1 % of the iteration) and the mode
// is not deterministic; returns whether it does.  An inner iteration takes 52.4 instead of 55.6 us at 16x128, and with the
// first step fused as well 69.7 instead of 72.7 at 32x256.
struct RzOut {
  const double* r = nullptr;
  const double* yy = nullptr;
  double* out = nullptr;
};
bool mg_apply(Ctx& c, const double* b, double* x, const MGOptions& o, bool first_done = false,
              const RzOut* rz = nullptr);
bool mg_apply_f(Ctx& c, const float* b, float* x, const MGOptions& o, bool first_done = false,
                const RzOut* rz = nullptr);
// The fine level's first smoother step from x = 0 for b: r = b, d = coef[0] D^-1 b,
// x = d, for a kernel that has b in registers anyway.  On fine levels with
// stencils only: a launch of 2 us is 3 % of an inner iteration at 32x256, while
// on larger levels the step is as fast in a launch of its own (64x512: 116.7
// fused, 116.4 us apart).
template <typename T>
struct FirstStep {
  const T* dinv = nullptr;   // null: the cycle takes the step itself
  T *r = nullptr, *d = nullptr, *x = nullptr;
  const double* coef = nullptr;
};
template <typename T>
FirstStep<T> mg_first_step(Ctx& c, T* x, const MGOptions& o);
template <typename T>
void launch_first_step(Ctx& c, const T* b, const FirstStep<T>& f);

// The small levels as one thread-block-cluster kernel (mgtail.cu): first level
// it covers, and its launcher (V-cycle of levels l0.. with b, x of level l0).
size_t tail_start(const Ctx& c, const MGOptions& o);
template <typename T>
void launch_vcycle_tail(Ctx& c, size_t l0, const T* b, T* x, bool first_done, const MGOptions& o);

}  // namespace dp
