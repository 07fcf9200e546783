// Thermal diffusion step on the P2 annulus: solveDiffusion_threaded
// (src/ThermalDiffusion/AssemblerThermal.jl:1-57), backward Euler
//   (M + dt K) T_new = M T_old,  T = Ttop / Tbot on the walls,
// with M = rho Cp mass and K the conduction matrix of assemble_element!
// (:114-226; 7-point rule, the element's curved inverse Jacobian).  The
// reference's force vector never reaches the system (the function returns
// before update_force_vector!), so neither does one here.
//
// Layout: the element blocks A_e = M_e + dt K_e (symmetric 6x6, 21 packed
// upper entries) entry-major, 168 B per element, in lattice order; the free
// nodes are all but the two walls (lattice radial index 0 and 2 ncr), found
// from the node index, so no index list is stored.
//
// k_th_assemble (one thread per element, FP64): A_e, diag(A) and b = M T_old
// - A T_bc by atomics (T_bc: the wall values, zero inside).  The solve is
// Jacobi-preconditioned CG (the matrix is SPD; the reference runs
// unpreconditioned GMRES) with the reference's stopping test ||r|| <= atol +
// rtol ||b|| (Krylov.jl's defaults sqrt(eps)), captured once per context as a
// CUDA graph whose WHILE node is continued or ended by the last block of the
// update kernel.  An iteration is two launches: k_th_apply forms p = z + beta p
// while it gathers it (p alternates between two buffers), q += A p and p.q;
// k_th_update x, r, z, beta, the stop test, and q = 0 for the next one.  A pass
// of a WHILE body costs ~10 us of its own, so a body holds kThUnroll
// iterations; those after the stopping test return at once.
// Gathering rows of A per node instead of elements (no atomics, 92 instead of 84
// bytes of matrix per node) measured 16-20 us per apply at 128x1024 against 9:
// each neighbour value is fetched 2 x 11.5 times instead of 2 x 3.
#include "kernels.cuh"
#include "reduce.cuh"

namespace dp {

// scalar-table slots of the thermal loop
enum ThSlot { TH_RZ = 48, TH_ALPHA = 50, TH_BETA = 51, TH_RR = 52, TH_TOL2 = 53, TH_IT = 54,
              TH_ITMAX = 55, TH_BB = 56, TH_RZN = 57, TH_STOP = 58 };

__constant__ double c_w7[7];  // 7-point weights x 0.5 (Quadrature.jl:109-138)

static void upload_thermal_constants() {
  const double w1 = (155.0 - std::sqrt(15.0)) / 1200.0, w2 = (155.0 + std::sqrt(15.0)) / 1200.0;
  const double w[7] = {0.5 * 0.225, 0.5 * w1, 0.5 * w1, 0.5 * w1, 0.5 * w2, 0.5 * w2, 0.5 * w2};
  DP_CUDA(cudaMemcpyToSymbol(c_w7, w, sizeof(w)));
}

constexpr int kThPack = 21;

__device__ __forceinline__ bool th_fixed(int64_t n, int64_t A, int amax, int heated) {
  const int a = (int)(n % A);
  return a == amax || (heated && a == 0);
}

struct ThAsmArgs {
  const double* theta_lat;
  const double* r_lat;
  const double* rho;   // nodal density, reference numbering
  const double* Told;  // reference numbering
  double* Ae;          // 21 x nel
  double* diag;        // nnod
  double* b;           // nnod
  double K, Cp, dt, Ttop, Tbot;
  int nel, ncr, nct, A, B, heated;
};

// prescribed value of a node on a wall, 0 inside
__device__ __forceinline__ double th_wall(int a, int amax, int heated, double Ttop, double Tbot) {
  return a == amax ? Ttop : ((heated && a == 0) ? Tbot : 0.0);
}

__global__ void __launch_bounds__(128) k_th_assemble(ThAsmArgs p) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= p.nel) return;
  int nd[6], nref[6];
  element_nodes_mg(e, p.ncr, p.A, p.B, nd);
  element_ref_nodes(e, p.ncr, p.nct, nref);
  double th[3], rr[3], rho[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    th[k] = p.theta_lat[nd[k]];
    rr[k] = p.r_lat[nd[k]];
    rho[k] = p.rho[nref[k]];
  }
  {
    const double PI = 3.14159265358979323846;
    const double d1 = fabs(th[0] - th[1]), d2 = fabs(th[1] - th[2]), d3 = fabs(th[2] - th[0]);
    if ((d1 + d2 + d3) > PI) {
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (th[k] < PI) th[k] += 2.0 * PI;
    }
  }
  // J = dN3ds * [theta r]: rows (dN/dxi, dN/deta) = (-1, 1, 0), (-1, 0, 1)
  const double J1 = -th[0] + th[1], J2 = -th[0] + th[2], J3 = -rr[0] + rr[1], J4 = -rr[0] + rr[2];
  const double detJ = J1 * J4 - J2 * J3, invdet = 1.0 / detJ;
  const double R21 = rr[1] - rr[0], R31 = rr[2] - rr[0];
  const double T31 = th[2] - th[0], T21 = th[1] - th[0];
  double Ke[kThPack], Me[kThPack];
#pragma unroll
  for (int k = 0; k < kThPack; ++k) Ke[k] = Me[k] = 0.0;
  for (int ip = 0; ip < 7; ++ip) {
    const double th_ip = th[0] * c_N3s[ip][0] + th[1] * c_N3s[ip][1] + th[2] * c_N3s[ip][2];
    const double r_ip = rr[0] * c_N3s[ip][0] + rr[1] * c_N3s[ip][1] + rr[2] * c_N3s[ip][2];
    const double rho_ip = rho[0] * c_N3s[ip][0] + rho[1] * c_N3s[ip][1] + rho[2] * c_N3s[ip][2];
    double s, c;
    sincos(th_ip, &s, &c);
    const double cr = c / r_ip, sr = s / r_ip;
    const double a11 = R31 * cr - T31 * s, a12 = -R21 * cr + T21 * s;
    const double a21 = -R31 * sr - T31 * c, a22 = R21 * sr + T21 * c;
    double dx[6], dz[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      dx[k] = (a11 * c_dNs[ip][0][k] + a12 * c_dNs[ip][1][k]) * invdet;
      dz[k] = (a21 * c_dNs[ip][0][k] + a22 * c_dNs[ip][1][k]) * invdet;
    }
    const double om = r_ip * detJ * c_w7[ip];
    const double wk = p.K * om, wm = om * rho_ip * p.Cp;
    int k = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
#pragma unroll
      for (int j = i; j < 6; ++j, ++k) {
        Ke[k] += wk * (dx[i] * dx[j] + dz[i] * dz[j]);
        Me[k] += wm * c_N6s[ip][i] * c_N6s[ip][j];
      }
    }
  }
  double to[6], tb[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    to[i] = p.Told[nref[i]];
    tb[i] = th_wall(nd[i] % p.A, 2 * p.ncr, p.heated, p.Ttop, p.Tbot);
  }
  double be[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const size_t st = (size_t)p.nel;
  int k = 0;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
#pragma unroll
    for (int j = i; j < 6; ++j, ++k) {
      const double a = Me[k] + p.dt * Ke[k];
      p.Ae[(size_t)k * st + e] = a;
      if (i == j) {
        atomicAdd(&p.diag[nd[i]], a);
        be[i] += Me[k] * to[i] - a * tb[i];
      } else {
        be[i] += Me[k] * to[j] - a * tb[j];
        be[j] += Me[k] * to[i] - a * tb[i];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) atomicAdd(&p.b[nd[i]], be[i]);
}

// p.q is added up in kThSlots scalars (a warp each, by index) that the update sums.
// kThUnroll is even, so which of the two p buffers an iteration of the body
// reads is known when it is captured.
constexpr int kThSlots = 128, kThUnroll = 4;
struct ThVecs {
  const double* Ae;
  const double* diag;
  double *x, *r, *z, *q, *slots;
  double *po, *pn;   // p before and after the iteration
};

// p' = z + beta p, q += A p' and p'.q over elements.  The type-0 element of a cell
// also stores p' for the cell's 2x2 nodes (the outer wall's nodes are fixed: p
// stays 0 there).
__global__ void __launch_bounds__(128) k_th_apply(ThVecs v, const double* scal, int nel, int ncr, int A, int B) {
  grid_dep_launch();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = e < nel;
  const int ec = live ? e : nel - 1;
  double a[kThPack];   // constant during the step: fetched before the wait
#pragma unroll
  for (int k = 0; k < kThPack; ++k) a[k] = ld_stream(v.Ae + (size_t)k * nel + ec);
  int nd[6];
  element_nodes_mg(ec, ncr, A, B, nd);
  grid_dep_sync();
  const double stop = scal[TH_STOP], beta = scal[TH_BETA];
  double zv[6], xv[6], yv[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    zv[i] = v.z[nd[i]];
    xv[i] = v.po[nd[i]];
  }
  if (stop != 0.0) return;   // the same for the whole grid
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    xv[i] = zv[i] + beta * xv[i];
    yv[i] = 0.0;
  }
  int k = 0;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
#pragma unroll
    for (int j = i; j < 6; ++j, ++k) {
      yv[i] += a[k] * xv[j];
      if (j != i) yv[j] += a[k] * xv[i];
    }
  }
  double d = 0.0;
  if (live) {
#pragma unroll
    for (int i = 0; i < 6; ++i) d += xv[i] * yv[i];
    if (!(e & 1)) {
#pragma unroll
      for (int i = 0; i < 6; ++i)
        if (i != 1 && i != 2) v.pn[nd[i]] = xv[i];   // local nodes 0, 3, 4, 5: the cell's own 2x2 block
    }
  }
  to_cell_order<double, 1>(yv, nd, ec);
  cell_scatter<double, 1, false>(yv, nd, v.q, e, nel, ncr);
  d = warp_sum(d);
  if ((threadIdx.x & 31) == 0) atomicAdd(&v.slots[(4 * blockIdx.x + (threadIdx.x >> 5)) % kThSlots], d);
}

// r = b (free), 0 (walls); z = r / diag; x = p = 0; sums r.z and b.b; p.q slots zeroed
__global__ void __launch_bounds__(kRedThreads) k_th_init(const double* __restrict__ b, ThVecs v, int64_t n, int64_t A,
                                                         int amax, int heated, double* scal, double* partial,
                                                         unsigned int* counter, double rtol, double atol, int itmax) {
  double s[2] = {0.0, 0.0};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const bool fx = th_fixed(i, A, amax, heated);
    const double ri = fx ? 0.0 : b[i];
    const double zi = fx ? 0.0 : ri / v.diag[i];
    v.x[i] = 0.0;
    v.r[i] = ri;
    v.z[i] = zi;
    v.po[i] = 0.0;
    v.pn[i] = 0.0;
    v.q[i] = 0.0;
    s[0] += ri * zi;
    s[1] += ri * ri;
  }
  if (blockIdx.x == 0 && threadIdx.x < kThSlots) v.slots[threadIdx.x] = 0.0;
  double* outs[2] = {scal + TH_RZ, scal + TH_BB};
  if (grid_finish<2>(s, partial, counter, outs) && threadIdx.x == 0) {
    const double tol = atol + rtol * sqrt(scal[TH_BB]);
    scal[TH_TOL2] = tol * tol;
    scal[TH_RR] = scal[TH_BB];
    scal[TH_BETA] = 0.0;
    scal[TH_ALPHA] = 0.0;
    scal[TH_IT] = 0.0;
    scal[TH_STOP] = 0.0;
    scal[TH_ITMAX] = (double)itmax;
  }
}

// sets the loop's condition before its first pass
__global__ void k_th_start(cudaGraphConditionalHandle h, const double* scal) {
  grid_dep_wait();
  cudaGraphSetConditional(h, (scal[TH_RR] > scal[TH_TOL2] && scal[TH_ITMAX] >= 1.0) ? 1u : 0u);
}

// x += alpha p; r -= alpha q; z = r / diag; beta and the stop test.  Two nodes per
// thread and access (the node count is even), all loads issued first.
__global__ void __launch_bounds__(kRedThreads) k_th_update(ThVecs v, int64_t n, int A, int amax, int heated,
                                                           double* scal, double* partial, unsigned int* counter,
                                                           cudaGraphConditionalHandle h) {
  grid_dep_wait();
  if (scal[TH_STOP] != 0.0) return;   // the same for the whole grid
  double pq = 0.0;
#pragma unroll
  for (int k = 0; k < kThSlots / 32; ++k) pq += v.slots[(threadIdx.x & 31) + 32 * k];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) pq += __shfl_xor_sync(0xffffffffu, pq, o);
  const double alpha = scal[TH_RZ] / pq;
  const double* p = v.pn;
  double s[2] = {0.0, 0.0};
  for (int64_t i = 2 * (blockIdx.x * (int64_t)blockDim.x + threadIdx.x); i < n;
       i += 2 * (int64_t)gridDim.x * blockDim.x) {
    const double2 pv = *reinterpret_cast<const double2*>(p + i), qv = *reinterpret_cast<const double2*>(v.q + i);
    const double2 dv = *reinterpret_cast<const double2*>(v.diag + i);
    double2 xv = *reinterpret_cast<const double2*>(v.x + i), rv = *reinterpret_cast<const double2*>(v.r + i);
    double2 zv = make_double2(0.0, 0.0);
    const int a0 = (int)(i % A), a1 = a0 + 1 == A ? 0 : a0 + 1;
    if (!(a0 == amax || (heated && a0 == 0))) {
      xv.x += alpha * pv.x;
      rv.x -= alpha * qv.x;
      zv.x = rv.x / dv.x;
    }
    if (!(a1 == amax || (heated && a1 == 0))) {
      xv.y += alpha * pv.y;
      rv.y -= alpha * qv.y;
      zv.y = rv.y / dv.y;
    }
    *reinterpret_cast<double2*>(v.x + i) = xv;
    *reinterpret_cast<double2*>(v.r + i) = rv;
    *reinterpret_cast<double2*>(v.z + i) = zv;
    *reinterpret_cast<double2*>(v.q + i) = make_double2(0.0, 0.0);   // the next apply adds to it
    s[0] += rv.x * zv.x + rv.y * zv.y;
    s[1] += rv.x * rv.x + rv.y * rv.y;
  }
  double* outs[2] = {scal + TH_RZN, scal + TH_RR};
  if (!grid_finish<2>(s, partial, counter, outs)) return;
  // the last block: every other one has read the slots
  if (threadIdx.x < kThSlots) v.slots[threadIdx.x] = 0.0;
  if (threadIdx.x == 0) {
    scal[TH_ALPHA] = alpha;
    scal[TH_BETA] = scal[TH_RZN] / scal[TH_RZ];
    scal[TH_RZ] = scal[TH_RZN];
    const double it = scal[TH_IT] + 1.0;
    scal[TH_IT] = it;
    const double rr = scal[TH_RR];
    const bool go = isfinite(rr) && isfinite(alpha) && rr > scal[TH_TOL2] && it < scal[TH_ITMAX];
    if (!go) scal[TH_STOP] = 1.0;   // the body's remaining iterations return at once
    cudaGraphSetConditional(h, go ? 1u : 0u);
  }
}

// T (reference numbering) = x (free) or the prescribed value (walls)
__global__ void k_th_finish(const double* __restrict__ x, double* __restrict__ T, int n, int A, int ncr, int nct,
                            int heated, double Ttop, double Tbot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int b = i / A, a = i - b * A;
  T[ref_of_lattice(a, b, ncr, nct)] = x[i] + th_wall(a, 2 * ncr, heated, Ttop, Tbot);
}

// thermal work vectors, nnod each, after the 21 x nel element blocks and the slots
enum ThVec { TV_DIAG = 0, TV_B, TV_X, TV_R, TV_Z, TV_P0, TV_P1, TV_Q, TV_T, TV_RHO, TV_COUNT };

static double* th_slots(Ctx& c) { return c.th_buf + kThPack * c.fine.nel; }
static double* th_vec(Ctx& c, int k) { return th_slots(c) + kThSlots + (size_t)k * c.fine.nnod; }
static int64_t th_doubles(const Ctx& c) {
  return kThPack * c.fine.nel + kThSlots + (int64_t)TV_COUNT * c.fine.nnod;
}
// of the k-th iteration of a body
static ThVecs th_vecs(Ctx& c, int k) {
  return ThVecs{c.th_buf,         th_vec(c, TV_DIAG), th_vec(c, TV_X),  th_vec(c, TV_R), th_vec(c, TV_Z),
                th_vec(c, TV_Q), th_slots(c),        th_vec(c, k & 1 ? TV_P1 : TV_P0),
                th_vec(c, k & 1 ? TV_P0 : TV_P1)};
}
static void th_launch_apply(Ctx& c, int k, cudaStream_t s) {
  const Level& L = c.fine;
  klaunch(k_th_apply, (int)div_up(L.nel, 128), 128, 0, s, th_vecs(c, k), (const double*)c.scal, (int)L.nel, L.ncr,
          (int)L.A(), (int)L.B());
  DP_LAUNCH_CHECK();
}

static void th_emit_loop(Ctx& c, int heated) {
  const Level& L = c.fine;
  const int64_t n = L.nnod;
  const int amax = 2 * L.ncr;
  cudaGraphConditionalHandle h = new_handle(c.stream);
  klaunch(k_th_start, 1, 1, 0, c.stream, h, (const double*)c.scal);
  DP_LAUNCH_CHECK();
  cudaGraph_t body = add_while(c.stream, h);
  cudaStream_t aux = c.aux[0];
  DP_CUDA(cudaStreamBeginCaptureToGraph(aux, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
  for (int k = 0; k < kThUnroll; ++k) {
    th_launch_apply(c, k, aux);
    // a pair of nodes per thread, as long as the grid stays within the partial buffer
    klaunch(k_th_update, (int)std::min<int64_t>(kRedBlocks, div_up(n / 2, kRedThreads)), kRedThreads, 0, aux,
            th_vecs(c, k), n, (int)L.A(), amax, heated, c.scal, c.partial, c.counter, h);
  }
  DP_LAUNCH_CHECK();
  cudaGraph_t out = nullptr;
  DP_CUDA(cudaStreamEndCapture(aux, &out));
}

// Kernel timing: the apply on the last step's blocks and vectors, after the stop
// flag that the step left was taken down (the apply does not raise it; what it adds
// to q and the slots is zeroed by the next step).
void th_clear_stop(Ctx& c) { DP_CUDA(cudaMemsetAsync(c.scal + TH_STOP, 0, sizeof(double), c.stream)); }
void launch_th_apply_staged(Ctx& c) { th_launch_apply(c, 0, c.stream); }

}  // namespace dp

using namespace dp;

extern "C" void dp_default_thermal_opts(dp_thermal_opts* o) {
  if (!o) return;
  o->K = 3.3;
  o->Cp = 1.2e3;
  o->dt = 0.0;
  o->Ttop = 300.0;
  o->Tbot = 4000.0;
  o->rtol = 1.4901161193847656e-08;  // sqrt(eps), Krylov.jl's default
  o->atol = 1.4901161193847656e-08;
  o->heated = 1;
  o->itmax = 0;  // 0: the number of nodes (Krylov.jl's 2n cap for GMRES; CG needs far fewer)
}

extern "C" int dp_thermal_step(dp_ctx* h, const dp_thermal_opts* o, const double* rho_node, double* T,
                               int32_t* iterations, double* relres, int32_t mem) {
  if (!h) return DP_BAD_ARG;
  Ctx& c = h->c;
  return guarded(&c, [&] {
    DP_CUDA(cudaSetDevice(c.device));
    if (!o || !rho_node || !T) throw BadArg("null argument");
    if (!(o->dt >= 0.0) || !std::isfinite(o->dt)) throw BadArg("dt must be finite and >= 0");
    if (!(o->K >= 0.0) || !(o->Cp > 0.0)) throw BadArg("K must be >= 0 and Cp > 0");
    if (!(o->rtol >= 0.0) || !(o->atol >= 0.0)) throw BadArg("tolerances must be >= 0");
    if (o->itmax < 0) throw BadArg("itmax must be >= 0");
    const Level& L = c.fine;
    const int64_t nel = L.nel, nn = L.nnod;
    static bool uploaded[64] = {false};
    if (c.device < 0 || c.device >= 64 || !uploaded[c.device]) {
      upload_stress_constants();
      upload_rheology_constants();
      upload_thermal_constants();
      DP_CUDA(cudaDeviceSynchronize());  // the copies are on the default stream; ours does not wait on it
      if (c.device >= 0 && c.device < 64) uploaded[c.device] = true;
    }
    if (!c.th_buf) dalloc(&c.th_buf, th_doubles(c));
    const int heated = o->heated ? 1 : 0;
    const int amax = 2 * L.ncr;
    double* b = th_vec(c, TV_B);
    double* Tdev = in_place(c.device, T, mem) ? T : th_vec(c, TV_T);
    static_assert(TV_B == TV_DIAG + 1, "diag and b are zeroed together");
    DP_CUDA(cudaMemsetAsync(th_vec(c, TV_DIAG), 0, sizeof(double) * 2 * nn, c.stream));
    ThAsmArgs a;
    a.theta_lat = c.theta_lat; a.r_lat = c.r_lat;
    a.rho = staged(c, rho_node, th_vec(c, TV_RHO), nn, mem);
    a.Told = Tdev;
    if (Tdev != T) DP_CUDA(cudaMemcpyAsync(Tdev, T, sizeof(double) * nn, kind_in(mem), c.stream));
    a.Ae = c.th_buf; a.diag = th_vec(c, TV_DIAG); a.b = b; a.K = o->K; a.Cp = o->Cp; a.dt = o->dt; a.Ttop = o->Ttop; a.Tbot = o->Tbot;
    a.nel = (int)nel; a.ncr = L.ncr; a.nct = L.nct; a.A = (int)L.A(); a.B = (int)L.B(); a.heated = heated;
    ++g_klaunch;
    k_th_assemble<<<(int)div_up(nel, 128), 128, 0, c.stream>>>(a);
    DP_LAUNCH_CHECK();
    const int itmax = o->itmax > 0 ? o->itmax : (int)std::min<int64_t>(nn, INT32_MAX);
    ++g_klaunch;
    k_th_init<<<red_grid(nn), kRedThreads, 0, c.stream>>>(b, th_vecs(c, 0), nn, L.A(), amax, heated, c.scal, c.partial,
                                                        c.counter, o->rtol, o->atol, itmax);
    DP_LAUNCH_CHECK();
    // the CG loop: one graph per context and wall configuration
    if (!c.th_exec || c.th_heated != heated) {
      if (c.th_exec) {
        cudaGraphExecDestroy((cudaGraphExec_t)c.th_exec);
        c.th_exec = nullptr;
      }
      ensure_ctl(c);  // the capture streams of loop bodies
      cudaGraph_t g = nullptr;
      DP_CUDA(cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeRelaxed));
      try {
        PdlScope pdl(1);
        th_emit_loop(c, heated);
      } catch (...) {
        // leave the stream out of capture mode before reporting the error
        cudaGraph_t partial = nullptr;
        cudaStreamEndCapture(c.stream, &partial);
        if (partial) cudaGraphDestroy(partial);
        cudaGetLastError();
        throw;
      }
      DP_CUDA(cudaStreamEndCapture(c.stream, &g));
      cudaGraphExec_t ex = nullptr;
      DP_CUDA(cudaGraphInstantiate(&ex, g, 0));
      cudaGraphDestroy(g);
      c.th_exec = ex;
      c.th_heated = heated;
    }
    DP_CUDA(cudaGraphLaunch((cudaGraphExec_t)c.th_exec, c.stream));
    ++g_klaunch;
    k_th_finish<<<(int)div_up(nn, 256), 256, 0, c.stream>>>(th_vec(c, TV_X), Tdev, (int)nn, (int)L.A(), L.ncr, L.nct,
                                                          heated, o->Ttop, o->Tbot);
    DP_LAUNCH_CHECK();
    if (Tdev != T) DP_CUDA(cudaMemcpyAsync(T, Tdev, sizeof(double) * nn, kind_out(mem), c.stream));
    DP_CUDA(cudaMemcpyAsync(c.h_scal, c.scal, sizeof(double) * 64, cudaMemcpyDeviceToHost, c.stream));
    DP_CUDA(cudaStreamSynchronize(c.stream));
    const double it = c.h_scal[TH_IT];
    const double rel = c.h_scal[TH_BB] > 0.0 ? std::sqrt(c.h_scal[TH_RR] / c.h_scal[TH_BB]) : 0.0;
    if (iterations) *iterations = (int32_t)it;
    if (relres) *relres = rel;
    if (!std::isfinite(rel)) return (int)DP_BREAKDOWN;
    return (c.h_scal[TH_RR] > c.h_scal[TH_TOL2]) ? (int)DP_NOT_CONVERGED : (int)DP_OK;
  });
}
