// Strain-rate / stress post-processor: stress! (src/Stress/StressCalculation.jl:
// 23-249), called after each Stokes solve with the Cartesian velocity
// (MAIN.jl:241-243, nip = 7: MAIN.jl:94, :164).
//
// One thread per element (FP64).  Per 7-point IP: the curved inverse Jacobian
// of the (theta, r)-linear element (the same geometry as the assembly), the P2
// derivatives dN/dx, dN/dz, the strain rate (exx, ezz, exz = (dux/dz +
// duz/dx) / 2) and its second invariant, and the deviatoric stress with its
// invariant: isotropic eta (4/3, -2/3, 2) or, with a tensor, the reference's
// anisotropic formula (:219-233, including its factors: eta13 * exz in tau_xx,
// eta23 * 2 exz in tau_zz, eta33 * exz in tau_xz).  Outputs are the reference's
// nel x 7 matrices (element fastest), eight of them in a row.
#include "kernels.cuh"

namespace dp {

__constant__ double c_N3s[7][3];     // linear N3 at the 7 IPs (Quadrature.jl:109-138)
__constant__ double c_dNs[7][2][6];  // P2 dN/d(r, s) at the 7 IPs (sf_dN_tri6, :287-307)

static void upload_stress_constants() {
  double N3[7][3], dN[7][2][6];
  const double g1 = (6.0 - std::sqrt(15.0)) / 21.0, g2 = (6.0 + std::sqrt(15.0)) / 21.0;
  const double ip[7][2] = {{1.0 / 3.0, 1.0 / 3.0}, {1.0 - 2.0 * g1, g1}, {g1, 1.0 - 2.0 * g1}, {g1, g1},
                           {1.0 - 2.0 * g2, g2},   {g2, 1.0 - 2.0 * g2}, {g2, g2}};
  for (int q = 0; q < 7; ++q) {
    const double r = ip[q][0], s = ip[q][1], t = 1.0 - r - s;
    N3[q][0] = t; N3[q][1] = r; N3[q][2] = s;
    const double dr[6] = {-(4.0 * t - 1.0), 4.0 * r - 1.0, 0.0, 4.0 * (t - r), 4.0 * s, -4.0 * s};
    const double ds[6] = {-(4.0 * t - 1.0), 0.0, 4.0 * s - 1.0, -4.0 * r, 4.0 * r, 4.0 * (t - s)};
    for (int k = 0; k < 6; ++k) {
      dN[q][0][k] = dr[k];
      dN[q][1][k] = ds[k];
    }
  }
  DP_CUDA(cudaMemcpyToSymbol(c_N3s, N3, sizeof(N3)));
  DP_CUDA(cudaMemcpyToSymbol(c_dNs, dN, sizeof(dN)));
}

// The caller's arrays: eta 7 columns of ld_eta, the six tensor fields 7 columns
// of ld_C each, out 56 columns of nel; U the Cartesian velocity in the reference
// numbering, interleaved (ux, uz).
struct StressArgs {
  const double* U;
  const double* theta_lat;
  const double* r_lat;
  const double* eta;
  const double* C[6];
  double* out;
  int64_t ld_eta, ld_C;
  int nel, ncr, nct, A, B, tensor, u16;   // u16: U is 16-byte aligned
};

// Reads and writes the caller's device arrays in place (host arrays are staged):
// at 256x2048 with a tensor 822 us per call when every array went through a
// staging copy and U through a permutation pass of its own, of which this
// kernel was 184 us.
__global__ void __launch_bounds__(128) k_stress(StressArgs p) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= p.nel) return;
  const int A = p.A, B = p.B;
  const double* __restrict__ theta_lat = p.theta_lat;
  const double* __restrict__ r_lat = p.r_lat;
  double ux[6], uz[6];
  {
    int m[6];
    element_ref_nodes(e, p.ncr, p.nct, m);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      if (p.u16) {
        const double2 v = reinterpret_cast<const double2*>(p.U)[m[k]];
        ux[k] = v.x;
        uz[k] = v.y;
      } else {
        ux[k] = p.U[2 * (size_t)m[k]];
        uz[k] = p.U[2 * (size_t)m[k] + 1];
      }
    }
  }
  int nd[6];
  element_nodes_mg(e, p.ncr, A, B, nd);
  // vertex coordinates + fixangles! (Utilities.jl:45-61)
  double th[3], rr[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    th[k] = theta_lat[nd[k]];
    rr[k] = r_lat[nd[k]];
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
  const double Jt0 = -th[0] + th[1], Jt1 = -th[0] + th[2];
  const double Jr0 = -rr[0] + rr[1], Jr1 = -rr[0] + rr[2];
  const double invdet = 1.0 / (Jt0 * Jr1 - Jt1 * Jr0);
  const double R21 = rr[1] - rr[0], R31 = rr[2] - rr[0];
  const double T31 = th[2] - th[0], T21 = th[1] - th[0];
  const size_t st = (size_t)p.nel;
  for (int ip = 0; ip < 7; ++ip) {
    const double th_ip = th[0] * c_N3s[ip][0] + th[1] * c_N3s[ip][1] + th[2] * c_N3s[ip][2];
    const double r_ip = rr[0] * c_N3s[ip][0] + rr[1] * c_N3s[ip][1] + rr[2] * c_N3s[ip][2];
    double s, c;
    sincos(th_ip, &s, &c);
    const double cr = c / r_ip, sr = s / r_ip;
    const double a11 = R31 * cr - T31 * s, a12 = -R21 * cr + T21 * s;
    const double a21 = -R31 * sr - T31 * c, a22 = R21 * sr + T21 * c;
    double exx = 0.0, ezz = 0.0, duxdz = 0.0, duzdx = 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const double dx = (a11 * c_dNs[ip][0][k] + a12 * c_dNs[ip][1][k]) * invdet;
      const double dz = (a21 * c_dNs[ip][0][k] + a22 * c_dNs[ip][1][k]) * invdet;
      exx += dx * ux[k];
      ezz += dz * uz[k];
      duxdz += dz * ux[k];
      duzdx += dx * uz[k];
    }
    const double exz = 0.5 * (duxdz + duzdx);
    const double et = __ldg(p.eta + ip * p.ld_eta + e);
    double txx, tzz, txz;
    if (p.tensor) {
      const size_t i = (size_t)(ip * p.ld_C + e);
      const double c11 = __ldg(p.C[0] + i) * et, c33 = __ldg(p.C[1] + i) * et, c55 = __ldg(p.C[2] + i) * et;
      const double c13 = __ldg(p.C[3] + i) * et, c15 = __ldg(p.C[4] + i) * et, c35 = __ldg(p.C[5] + i) * et;
      const double pa = -exx / 3.0 + 2.0 * ezz / 3.0, pb = 2.0 * exx / 3.0 - ezz / 3.0;
      txx = c13 * pa + c11 * pb + c15 * exz;
      tzz = c33 * pa + c13 * pb + c35 * 2.0 * exz;
      txz = c35 * pa + c15 * pb + c55 * exz;
    } else {
      txx = et * (4.0 / 3.0 * exx - 2.0 / 3.0 * ezz);
      tzz = et * (-2.0 / 3.0 * exx + 4.0 / 3.0 * ezz);
      txz = et * 2.0 * exz;
    }
    double* o = p.out + (size_t)ip * st + e;
    const size_t blk = 7 * st;
    o[0 * blk] = exx;
    o[1 * blk] = ezz;
    o[2 * blk] = exz;
    o[3 * blk] = sqrt(0.5 * (exx * exx + ezz * ezz) + exz * exz);
    o[4 * blk] = txx;
    o[5 * blk] = tzz;
    o[6 * blk] = txz;
    o[7 * blk] = sqrt(0.5 * (txx * txx + tzz * tzz) + txz * txz);
  }
}

static StressArgs stress_args(Ctx& c, bool tensor) {
  StressArgs a{};
  a.theta_lat = c.theta_lat; a.r_lat = c.r_lat;
  a.nel = (int)c.fine.nel; a.ncr = c.fine.ncr; a.nct = c.fine.nct; a.A = (int)c.fine.A(); a.B = (int)c.fine.B();
  a.tensor = tensor ? 1 : 0;
  return a;
}
static void launch_stress(Ctx& c, StressArgs a) {
  a.u16 = aligned16(a.U) ? 1 : 0;
  ++g_klaunch;
  k_stress<<<(int)div_up(a.nel, 128), 128, 0, c.stream>>>(a);
  DP_LAUNCH_CHECK();
}
// the staging buffer: eta 7, tensor 42, out 56 columns
static StressArgs staged_stress_args(Ctx& c, bool tensor) {
  const int64_t nel = c.fine.nel;
  if (!c.stress_buf) dalloc(&c.stress_buf, (7 + 42 + 56) * nel);
  StressArgs a = stress_args(c, tensor);
  a.U = (const double*)c.work[W_UC];
  a.eta = c.stress_buf;
  for (int f = 0; f < 6; ++f) a.C[f] = c.stress_buf + (7 + 7 * f) * nel;
  a.out = c.stress_buf + 49 * nel;
  a.ld_eta = a.ld_C = nel;
  return a;
}

// k_stress on the inputs of the last staged call (kernel timing)
void launch_stress_staged(Ctx& c, bool tensor) { launch_stress(c, staged_stress_args(c, tensor)); }

}  // namespace dp

using namespace dp;

extern "C" int dp_stress(dp_ctx* h, const double* Ucart, const double* eta_ip, int64_t ld_eta,
                         const double* const* C6, int64_t ld_C, double* out, int32_t mem) {
  if (!h) return DP_BAD_ARG;
  Ctx& c = h->c;
  return guarded(&c, [&] {
    DP_CUDA(cudaSetDevice(c.device));
    if (!Ucart || !eta_ip || !out) throw BadArg("null argument");
    const int64_t nel = c.fine.nel, nn = c.fine.nnod;
    if (ld_eta < nel || (C6 && ld_C < nel)) throw BadArg("leading dimension below nel");
    static bool uploaded[64] = {false};
    if (c.device < 0 || c.device >= 64 || !uploaded[c.device]) {
      upload_stress_constants();
      DP_CUDA(cudaDeviceSynchronize());  // the copies are on the default stream; ours does not wait on it
      if (c.device >= 0 && c.device < 64) uploaded[c.device] = true;
    }
    if (C6)
      for (int f = 0; f < 6; ++f)
        if (!C6[f]) throw BadArg("null tensor field");
    bool dev = in_place(c.device, out, mem) && in_place(c.device, Ucart, mem) && in_place(c.device, eta_ip, mem) &&
               !overlap(out, 56 * nel, Ucart, 2 * nn) && !overlap(out, 56 * nel, eta_ip, 6 * ld_eta + nel);
    for (int f = 0; C6 && f < 6; ++f)
      dev = dev && in_place(c.device, C6[f], mem) && !overlap(out, 56 * nel, C6[f], 6 * ld_C + nel);
    if (dev) {
      StressArgs a = stress_args(c, C6 != nullptr);
      a.U = Ucart; a.eta = eta_ip; a.out = out;
      a.ld_eta = ld_eta; a.ld_C = ld_C;
      for (int f = 0; C6 && f < 6; ++f) a.C[f] = C6[f];
      launch_stress(c, a);
    } else {
      const StressArgs a = staged_stress_args(c, C6 != nullptr);
      // nel x 7 column-major (element fastest) -> 7 contiguous columns
      DP_CUDA(cudaMemcpy2DAsync((void*)a.eta, sizeof(double) * nel, eta_ip, sizeof(double) * ld_eta,
                                sizeof(double) * nel, 7, kind_in(mem), c.stream));
      for (int f = 0; C6 && f < 6; ++f)
        DP_CUDA(cudaMemcpy2DAsync((void*)a.C[f], sizeof(double) * nel, C6[f], sizeof(double) * ld_C,
                                  sizeof(double) * nel, 7, kind_in(mem), c.stream));
      DP_CUDA(cudaMemcpyAsync((void*)a.U, Ucart, sizeof(double) * 2 * nn, kind_in(mem), c.stream));
      c.stress_staged = true;
      c.stress_tensor = C6 != nullptr;
      launch_stress(c, a);
      DP_CUDA(cudaMemcpyAsync(out, a.out, sizeof(double) * 56 * nel, kind_out(mem), c.stream));
    }
    DP_CUDA(cudaStreamSynchronize(c.stream));
    return (int)DP_OK;
  });
}
