// Per-IP viscosity update, Arrhenius law with Drucker-Prager plasticity:
// getviscosity!(::Arrhenius, T, P, epsII, tauII, e2n, r) (src/Rheology/
// Rheology.jl:348-403), the producer of the eta.ip the Stokes assembly reads.
//
// One thread per element, 7-point IPs (Quadrature.jl:109-138): T_ip and the
// radius z_ip by the P2 shape functions, P_ip by the linear ones at the three
// vertices plus |min P| (a device reduction), a depth factor lambda (1e1
// between max r - 2780 km and max r - 660 km, 1e-3 below, 1e0 above), eta_TP =
// clamp(lambda eta0 exp((Ea + P Va) / (R T) - Ea / (R T0)), 1e18, 1e25)
// (getviscosity :171-173).  Where cohesion, friction angle and epsII are all
// non-zero the plastic branch applies: yield stress cosd(phi) C + sind(phi) P
// (druckerPrager :338-344) and, if it is below tauII, eta = clamp(tau_y /
// (2 epsII), 1e18, 1e25); otherwise the previous eta is kept, as the
// reference does.  eta is read and written in place.
#include "kernels.cuh"
#include "reduce.cuh"

namespace dp {

constexpr int S_MINP = 40, S_MAXR = 41;  // scalar-table slots of the two reductions

__constant__ double c_N6s[7][6];  // P2 N at the 7 IPs (sf_N_tri6, Quadrature.jl:264-285)

static void upload_rheology_constants() {
  double N6[7][6];
  const double g1 = (6.0 - std::sqrt(15.0)) / 21.0, g2 = (6.0 + std::sqrt(15.0)) / 21.0;
  const double ip[7][2] = {{1.0 / 3.0, 1.0 / 3.0}, {1.0 - 2.0 * g1, g1}, {g1, 1.0 - 2.0 * g1}, {g1, g1},
                           {1.0 - 2.0 * g2, g2},   {g2, 1.0 - 2.0 * g2}, {g2, g2}};
  for (int q = 0; q < 7; ++q) {
    const double r = ip[q][0], s = ip[q][1], t = 1.0 - r - s;
    const double n[6] = {t * (2.0 * t - 1.0), r * (2.0 * r - 1.0), s * (2.0 * s - 1.0),
                         4.0 * r * t, 4.0 * r * s, 4.0 * s * t};
    for (int k = 0; k < 6; ++k) N6[q][k] = n[k];
  }
  DP_CUDA(cudaMemcpyToSymbol(c_N6s, N6, sizeof(N6)));
}

// |min P| over the vertices and max r over the nodes, in one launch: the last
// block to arrive reduces the per-block values (a second launch of one thread
// over the 1184 pairs took 80 us).
__global__ void __launch_bounds__(kRedThreads) k_minmax(const double* __restrict__ P, int64_t np,
                                                        const double* __restrict__ r, int64_t nn, double* partial,
                                                        unsigned int* counter, double* scal) {
  __shared__ double smn[kRedThreads / 32], smx[kRedThreads / 32];
  __shared__ bool last;
  double mn = INFINITY, mx = -INFINITY;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x)
    mn = fmin(mn, P[i]);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nn; i += (int64_t)gridDim.x * blockDim.x)
    mx = fmax(mx, r[i]);
  auto block_minmax = [&]() {   // in thread 0
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn = fmin(mn, __shfl_down_sync(0xffffffffu, mn, o));
      mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
      smn[threadIdx.x >> 5] = mn;
      smx[threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < kRedThreads / 32; ++w) {
        mn = fmin(mn, smn[w]);
        mx = fmax(mx, smx[w]);
      }
    }
  };
  block_minmax();
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = mn;
    partial[gridDim.x + blockIdx.x] = mx;
    __threadfence();
    last = atomicInc(counter, gridDim.x) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  mn = INFINITY;
  mx = -INFINITY;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
    mn = fmin(mn, ((volatile double*)partial)[b]);
    mx = fmax(mx, ((volatile double*)partial)[gridDim.x + b]);
  }
  block_minmax();
  if (threadIdx.x == 0) {
    scal[S_MINP] = fabs(mn);
    scal[S_MAXR] = mx;
    *counter = 0;
  }
}

struct ArrheniusArgs {
  double eta0, R, Ea, Va, T0, sphi, cphi, phi;
};

// T, r (nodes) and P (vertices): reference numbering.  epsII, tauII, coh, eta:
// nel x 7 element-fastest.  All of them the caller's own arrays when they are on
// the device.
__global__ void __launch_bounds__(128) k_viscosity_arrhenius(const double* __restrict__ T, const double* __restrict__ P,
                                                             const double* __restrict__ r,
                                                             const double* __restrict__ epsII,
                                                             const double* __restrict__ tauII,
                                                             const double* __restrict__ coh, double* eta,
                                                             const double* scal, ArrheniusArgs law, int nel, int ncr,
                                                             int nct) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nel) return;
  int nd[6];
  element_ref_nodes(e, ncr, nct, nd);
  double Te[6], re[6], Pe[3];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    Te[k] = T[nd[k]];
    re[k] = r[nd[k]];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) Pe[k] = P[nd[k]];   // vertices are the first reference numbers
  const double minP = scal[S_MINP], maxr = scal[S_MAXR];
  const size_t st = (size_t)nel;
  for (int ip = 0; ip < 7; ++ip) {
    double T_ip = 0.0, z_ip = 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      T_ip += Te[k] * c_N6s[ip][k];
      z_ip += re[k] * c_N6s[ip][k];
    }
    const double P_ip = Pe[0] * c_N3s[ip][0] + Pe[1] * c_N3s[ip][1] + Pe[2] * c_N3s[ip][2] + minP;
    const double lam = z_ip < maxr - 2780e3 ? 1e-3 : (z_ip > maxr - 660e3 ? 1e0 : 1e1);
    const double etaTP =
        fmin(fmax(lam * law.eta0 * exp((law.Ea + P_ip * law.Va) / law.R / T_ip - law.Ea / law.R / law.T0), 1e18), 1e25);
    const size_t i = (size_t)ip * st + e;
    const double e2 = epsII[i], c = coh[i];
    if (c > 0.0 && law.phi > 0.0 && e2 != 0.0) {
      const double tau_y = law.cphi * c + law.sphi * P_ip;
      if (tau_y < tauII[i]) eta[i] = fmax(1e18, fmin(1e25, 0.5 * tau_y / e2));
    } else {
      eta[i] = etaTP;
    }
  }
}

static ArrheniusArgs last_law(const Ctx& c) {
  ArrheniusArgs a;
  a.eta0 = c.rheo_law[0]; a.R = c.rheo_law[1]; a.Ea = c.rheo_law[2]; a.Va = c.rheo_law[3];
  a.T0 = c.rheo_law[4]; a.sphi = c.rheo_law[5]; a.cphi = c.rheo_law[6]; a.phi = c.rheo_law[7];
  return a;
}
static void launch_viscosity(Ctx& c, const double* T, const double* P, const double* r, const double* e2,
                             const double* t2, const double* co, double* et) {
  const int nel = (int)c.fine.nel;
  ++g_klaunch;
  k_viscosity_arrhenius<<<(int)div_up(nel, 128), 128, 0, c.stream>>>(T, P, r, e2, t2, co, et, c.scal, last_law(c), nel,
                                                                      c.fine.ncr, c.fine.nct);
  DP_LAUNCH_CHECK();
}
// the staging buffer: epsII, tauII, cohesion, eta (7 columns each), T, P, r
static double* rheo_staging(Ctx& c) {
  if (!c.rheo_buf) dalloc(&c.rheo_buf, 28 * c.fine.nel + 3 * c.fine.nnod);
  return c.rheo_buf;
}

// k_viscosity_arrhenius on the inputs of the last staged call, with the last
// call's law and extremes (kernel timing; eta is updated in place, and a second
// pass over it writes the same values).
void launch_viscosity_staged(Ctx& c) {
  const int64_t nel = c.fine.nel, nn = c.fine.nnod;
  double* e2 = rheo_staging(c);
  double* Ts = e2 + 28 * nel;
  launch_viscosity(c, Ts, Ts + nn, Ts + 2 * nn, e2, e2 + 7 * nel, e2 + 14 * nel, e2 + 21 * nel);
}

}  // namespace dp

using namespace dp;

extern "C" int dp_viscosity_arrhenius(dp_ctx* h, const dp_arrhenius* law, const double* T_node, const double* P_vertex,
                                      int64_t nvert, const double* r_node, const double* epsII, const double* tauII,
                                      const double* cohesion, double* eta_ip, int32_t mem) {
  if (!h) return DP_BAD_ARG;
  Ctx& c = h->c;
  return guarded(&c, [&] {
    DP_CUDA(cudaSetDevice(c.device));
    if (!law || !T_node || !P_vertex || !r_node || !epsII || !tauII || !cohesion || !eta_ip)
      throw BadArg("null argument");
    const int64_t nel = c.fine.nel, nn = c.fine.nnod;
    const int64_t nv = (int64_t)(c.fine.ncr + 1) * c.fine.nct;
    if (nvert != nv) throw BadArg("P_vertex must hold the " + std::to_string(nv) + " vertex values");
    if (!(law->T0 > 0.0) || !(law->R > 0.0)) throw BadArg("T0 and R must be positive");
    static bool uploaded[64] = {false};
    if (c.device < 0 || c.device >= 64 || !uploaded[c.device]) {
      upload_rheology_constants();
      upload_stress_constants();
      DP_CUDA(cudaDeviceSynchronize());  // the copies are on the default stream; ours does not wait on it
      if (c.device >= 0 && c.device < 64) uploaded[c.device] = true;
    }
    bool dev = in_place(c.device, eta_ip, mem);
    auto readable = [&](const double* a, int64_t n) {
      dev = dev && in_place(c.device, a, mem) && !overlap(eta_ip, 7 * nel, a, n);
    };
    readable(T_node, nn);
    readable(P_vertex, nv);
    readable(r_node, nn);
    for (const double* a : {epsII, tauII, cohesion}) readable(a, 7 * nel);
    const double *T = T_node, *P = P_vertex, *r = r_node, *e2 = epsII, *t2 = tauII, *co = cohesion;
    double* et = eta_ip;
    if (!dev) {
      double* s = rheo_staging(c);
      auto up = [&](double* dst, const double* src, int64_t n) {
        DP_CUDA(cudaMemcpyAsync(dst, src, sizeof(double) * n, kind_in(mem), c.stream));
        return dst;
      };
      e2 = up(s, epsII, 7 * nel);
      t2 = up(s + 7 * nel, tauII, 7 * nel);
      co = up(s + 14 * nel, cohesion, 7 * nel);
      et = up(s + 21 * nel, eta_ip, 7 * nel);
      T = up(s + 28 * nel, T_node, nn);
      P = up(s + 28 * nel + nn, P_vertex, nv);
      r = up(s + 28 * nel + 2 * nn, r_node, nn);
      c.rheo_staged = true;
    }
    ++g_klaunch;
    k_minmax<<<(int)std::min<int64_t>(kRedBlocks, div_up(nn, 4 * kRedThreads)), kRedThreads, 0, c.stream>>>(
        P, nv, r, nn, c.partial, c.counter, c.scal);
    DP_LAUNCH_CHECK();
    ArrheniusArgs a;
    a.eta0 = law->eta0; a.R = law->R; a.Ea = law->Ea; a.Va = law->Va; a.T0 = law->T0; a.phi = law->phi_deg;
    a.sphi = std::sin(law->phi_deg * (3.14159265358979323846 / 180.0));
    a.cphi = std::cos(law->phi_deg * (3.14159265358979323846 / 180.0));
    const double keep[8] = {a.eta0, a.R, a.Ea, a.Va, a.T0, a.sphi, a.cphi, a.phi};
    for (int i = 0; i < 8; ++i) c.rheo_law[i] = keep[i];
    launch_viscosity(c, T, P, r, e2, t2, co, et);
    if (!dev) DP_CUDA(cudaMemcpyAsync(eta_ip, et, sizeof(double) * 7 * nel, kind_out(mem), c.stream));
    DP_CUDA(cudaStreamSynchronize(c.stream));
    return (int)DP_OK;
  });
}
