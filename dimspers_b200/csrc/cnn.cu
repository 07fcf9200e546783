// Learned initial guess for the Schur PCG: a small convolutional network on
// the polar grid of the half-resolution mesh's vertices (nrg = ncr/2 + 1
// radial x ntg = nct/2 angular points, periodic in theta), with hand-written
// forward, backward and Adam kernels.
//
// Network: L dilated 3x3 convolutions (zero padding in r, periodic in theta),
// ReLU after every layer but the last; inputs 4 channels (buoyancy rho,
// log10 eta, cos 2phi, sin 2phi of the director), output 1 channel: the
// pressure divided by g (Stokes is linear in the body force, so P/g does not
// depend on the Rayleigh number).  Activations are [batch][channel][r][theta]
// (theta fastest), FP32.  Forward pass and data gradient are implicit GEMMs on
// the tensor cores (BF16 operands, FP32 accumulation) or, on request and for
// grids whose theta size is not a multiple of 16, FP32 CUDA-core convolutions;
// the weight gradient is FP32 either way.
//
// The predicted grid pressure is prolongated bilinearly to the pressure DOFs
// (discontinuous: the element's vertex values; continuous: vertex values) and
// handed to dp_solve with use_guess = 2, which keeps it only if it lowers the
// initial Schur residual.
#include <cuda_bf16.h>

#include <cmath>
#include <vector>

namespace dp {

constexpr int kCnnMaxC = 32;
constexpr int kCnnMaxLayers = 12;

struct Cnn {
  int nrg = 0, ntg = 0, C = 16, L = 6, cin = 4, device = 0;
  int bf16 = 1;                 // 1: BF16 tensor-core convolutions (FP32 accumulate), 0: FP32 CUDA cores
  __nv_bfloat16* wk = nullptr;  // BF16 B operands of every layer, forward then data gradient (refreshed with the weights)
  std::vector<int64_t> wkoff;   // per layer: forward, data gradient
  float* wpart = nullptr;       // partial sums of the weight gradient (in dbuf0's allocation)
  int dil[kCnnMaxLayers];
  int bmax = 0;
  cudaStream_t stream = nullptr;
  std::string err;
  // parameters: per layer W[cout][cin][3][3] then b[cout], concatenated
  std::vector<int64_t> woff, boff;
  int64_t nparam = 0;
  float* param = nullptr;
  float* grad = nullptr;
  float* adam_m = nullptr;
  float* adam_v = nullptr;
  int64_t step = 0;
  std::vector<float*> act;   // act[0] = input (external), act[l+1] = output of layer l
  float* dbuf0 = nullptr;    // gradient buffers (max size), one allocation
  float* dbuf1 = nullptr;
  double* partial = nullptr;
  unsigned int* counter = nullptr;
  double* loss = nullptr;
  double* h_loss = nullptr;
  int cin_of(int l) const { return l == 0 ? cin : C; }
  int cout_of(int l) const { return l == L - 1 ? 1 : C; }
  ~Cnn() {
    cudaFree(param); cudaFree(grad); cudaFree(adam_m); cudaFree(adam_v);
    for (size_t i = 1; i < act.size(); ++i) cudaFree(act[i]);
    cudaFree(dbuf0); cudaFree(partial); cudaFree(counter); cudaFree(loss); cudaFree(wk);
    cudaFreeHost(h_loss);
    if (stream) cudaStreamDestroy(stream);
  }
};

// ---- kernels -------------------------------------------------------------------
// Y[b][co][i][j] = b[co] + sum_ci sum_taps W[co][ci][ti][tj] X[b][ci][i+(ti-1)d][j+(tj-1)d]
template <int COUT>
__global__ void __launch_bounds__(256) k_conv_fwd(const float* __restrict__ X, const float* __restrict__ W,
                                                  const float* __restrict__ bias, float* __restrict__ Y, int cin,
                                                  int nrg, int ntg, int dil, int relu) {
  extern __shared__ float sw[];  // COUT * cin * 9 + COUT
  const int nw = COUT * cin * 9;
  for (int k = threadIdx.x; k < nw + COUT; k += blockDim.x) sw[k] = k < nw ? W[k] : bias[k - nw];
  __syncthreads();
  const int b = blockIdx.z, i = blockIdx.y;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= ntg) return;
  float acc[COUT];
#pragma unroll
  for (int co = 0; co < COUT; ++co) acc[co] = sw[nw + co];
  const int64_t plane = (int64_t)nrg * ntg;
  for (int ci = 0; ci < cin; ++ci) {
    const float* Xc = X + ((int64_t)b * cin + ci) * plane;
#pragma unroll
    for (int ti = 0; ti < 3; ++ti) {
      const int ii = i + (ti - 1) * dil;
      if (ii < 0 || ii >= nrg) continue;
#pragma unroll
      for (int tj = 0; tj < 3; ++tj) {
        int jj = j + (tj - 1) * dil;
        jj = ((jj % ntg) + ntg) % ntg;
        const float xv = Xc[(int64_t)ii * ntg + jj];
#pragma unroll
        for (int co = 0; co < COUT; ++co) acc[co] += sw[(co * cin + ci) * 9 + ti * 3 + tj] * xv;
      }
    }
  }
#pragma unroll
  for (int co = 0; co < COUT; ++co) {
    float v = acc[co];
    if (relu && v < 0.f) v = 0.f;
    Y[((int64_t)b * COUT + co) * plane + (int64_t)i * ntg + j] = v;
  }
}

// ---- BF16 tensor-core convolutions (mma.sync m16n8k16, FP32 accumulation) ----------
// The forward convolution and the data gradient are both implicit GEMMs over
// the grid points: out[p][n] = sum_tap sum_k in[k][p + s*tap] * B[tap][n][k],
// with s = +1 (forward: k = input channel, n = output channel) or s = -1 (data
// gradient: k = output channel, n = input channel).  One warp computes 16
// consecutive theta points of one row times all NT*8 output columns; the K
// loop runs over the 9 taps and blocks of 16 channels.  A fragments are
// gathered from the FP32 activations and rounded to BF16; the B operand is
// the layer's weights rounded to BF16, laid out [tap][n][k] with a row stride
// of kpad + 8 elements, so the k pairs read from shared memory by a warp fall
// in distinct banks.
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);   // .x (low half) = lo
  return *reinterpret_cast<const uint32_t*>(&v);
}

// D += A B for one 16x8x16 tile: A rows = grid points, columns = k; B = k x n.
// Fragment layout (PTX ISA, mma.m16n8k16 with .bf16): a[0] = (row g, k 2t..2t+1),
// a[1] = (row g+8, k 2t..2t+1), a[2] = (row g, k 2t+8..2t+9), a[3] = (row g+8,
// k 2t+8..2t+9); b0 = (k 2t..2t+1, col g), b1 = (k 2t+8..2t+9, col g); d[0..1] =
// (row g, col 2t..2t+1), d[2..3] = (row g+8, col 2t..2t+1), with g = lane/4,
// t = lane%4.
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm_x2(uint32_t& r0, uint32_t& r1, const void* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(a) : "memory");
}

// B operands of all layers: Bk[tap][n][k] (row stride kpad + 8) from
// W[co][ci][tap]; forward n = co, k = ci; data gradient n = ci, k = co.  Zero
// outside the layer.  blockIdx.y = 2 layer + direction.
struct WkArgs {
  int64_t w[kCnnMaxLayers], o[2 * kCnnMaxLayers];
  int cin[kCnnMaxLayers], cout[kCnnMaxLayers];
};
__global__ void k_conv_weights_bf16(const float* __restrict__ P, __nv_bfloat16* __restrict__ out, WkArgs a) {
  const int l = blockIdx.y >> 1, transpose = blockIdx.y & 1;
  const int cin = a.cin[l], cout = a.cout[l];
  const int nch = transpose ? cin : cout, kch = transpose ? cout : cin;
  const int npad = (nch + 7) / 8 * 8, kpad = (kch + 15) / 16 * 16, ks = kpad + 8;
  const float* W = P + a.w[l];
  __nv_bfloat16* Bk = out + a.o[blockIdx.y];
  const int total = 9 * npad * ks;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const int tap = idx / (npad * ks), rem = idx % (npad * ks), n = rem / ks, k = rem % ks;
    const int co = transpose ? k : n, ci = transpose ? n : k;
    float v = 0.f;
    if (k < kpad && co < cout && ci < cin) v = W[(co * cin + ci) * 9 + tap];
    Bk[idx] = __float2bfloat16_rn(v);
  }
}

// Columns of a row window of TJ grid points and the points d to either side that
// its taps need, as they are staged: one run where the shifted windows overlap
// (d < TJ), else three windows side by side.  Tap tj of point p is column
// p + tj * min(d, TJ).
__host__ __device__ inline int win_cols(int tj, int d) { return tj + 2 * (d < tj ? d : tj); }
__device__ __forceinline__ int win_point(int col, int j0, int tj, int d, int ntg) {
  int j = d < tj ? j0 - d + col : j0 + (col / tj - 1) * d + col % tj;
  j %= ntg;
  return j < 0 ? j + ntg : j;
}
// the points of a lane's columns lane, lane + 32, ... (the same for every row and
// channel of a window, so the divisions are done once per window)
template <int TJ>
struct LanePoints {
  static constexpr int kMax = 3 * TJ / 32;
  int j[kMax];
  __device__ __forceinline__ void set(int lane, int ncol, int j0, int d, int ntg) {
#pragma unroll
    for (int k = 0; k < kMax; ++k) j[k] = lane + 32 * k < ncol ? win_point(lane + 32 * k, j0, TJ, d, ntg) : -1;
  }
};

// out[b][n][i][j] = bias[n] + sum_tap sum_k X[b][k][i + s(ti-1)d][j + s(tj-1)d] Bk[tap][n][k]
// (zero rows outside [0, nrg), periodic in j), ReLU optional; with mask, zero
// where mask[b][n][i][j] <= 0 (the gradient through the ReLU of the layer
// below); with affine, v * scale + shift as two roundings.  ntg % 16 == 0.
// One CTA = 16 WARPS consecutive theta points of one row and all output columns.
// The three input rows are read once, coalesced, rounded to BF16 and kept in
// shared memory as [point][channel] (stride kpad + 8: ldmatrix without bank
// conflicts), so a rounding and a global read serve all taps and columns; the
// result leaves through shared memory in 16-byte rows.  Bound by the latency of
// the staging loads (16 in flight per thread).  The form that gathered the
// fragments from global memory took 30 us per layer (65 x 512, 32 channels,
// batch 1) and 100 us at batch 8.  The order of the accumulation (tap by tap,
// 16 channels at a time) is unchanged.
template <int NT, int WARPS>
struct ConvTile {
  static constexpr int kTj = 16 * WARPS, kOs = kTj + 4;
  static size_t smem(int kpad, int dil) {
    const size_t win = sizeof(__nv_bfloat16) * (kpad + 8) * 3 * (size_t)win_cols(kTj, dil);
    const size_t out = sizeof(float) * NT * 8 * kOs;
    return sizeof(__nv_bfloat16) * (kpad + 8) * 9 * NT * 8 + std::max(win, out);
  }
};

template <int NT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) k_conv_tc(const float* __restrict__ X,
                                                        const __nv_bfloat16* __restrict__ Bk,
                                                        const float* __restrict__ bias,
                                                        const float* __restrict__ mask, float* __restrict__ Y,
                                                        int kch, int kpad, int nch, int nrg, int ntg, int dil, int sgn,
                                                        int relu, int affine, float scale, float shift) {
  constexpr int TJ = ConvTile<NT, WARPS>::kTj, OS = ConvTile<NT, WARPS>::kOs;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ks = kpad + 8, ncol = win_cols(TJ, dil), step = dil < TJ ? dil : TJ;
  __nv_bfloat16* sb = reinterpret_cast<__nv_bfloat16*>(smem_raw);
  __nv_bfloat16* sx = sb + 9 * NT * 8 * ks;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.z, i = blockIdx.y, j0 = blockIdx.x * TJ;
  const int64_t plane = (int64_t)nrg * ntg;
  const float* Xb = X + (int64_t)b * kch * plane;
  // stage: an item is one row, 8 channels, 32 columns (a lane each); two items per round
  const int ng = kpad / 8, nkb = (ncol + 31) / 32, items = 3 * ng * nkb;
  const bool plain = dil < TJ && ntg >= TJ + dil;   // one wrap at most, no division
  for (int it0 = warp; it0 < items; it0 += 2 * WARPS) {
    float v[2][8];
    __nv_bfloat16* dst[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int it = it0 + h * WARPS, rg = it / nkb, col = lane + 32 * (it - rg * nkb);
      const int row = rg / ng, c0 = 8 * (rg - row * ng), ii = i + (row - 1) * dil;
      const bool ok = it < items && col < ncol && ii >= 0 && ii < nrg;
      int j = 0;
      if (plain) {
        j = j0 - dil + col;
        j += j < 0 ? ntg : 0;
        j -= j >= ntg ? ntg : 0;
      } else if (ok) {
        j = win_point(col, j0, TJ, dil, ntg);
      }
      const float* p = Xb + (int64_t)c0 * plane + (int64_t)ii * ntg + j;
#pragma unroll
      for (int c = 0; c < 8; ++c) v[h][c] = ok && c0 + c < kch ? p[(int64_t)c * plane] : 0.f;
      dst[h] = ok ? sx + ((int64_t)row * ncol + col) * ks + c0 : nullptr;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (!dst[h]) continue;
      uint4 o;
      o.x = pack_bf16(v[h][0], v[h][1]);
      o.y = pack_bf16(v[h][2], v[h][3]);
      o.z = pack_bf16(v[h][4], v[h][5]);
      o.w = pack_bf16(v[h][6], v[h][7]);
      *reinterpret_cast<uint4*>(dst[h]) = o;
    }
  }
  {
    const uint4* src = reinterpret_cast<const uint4*>(Bk);
    uint4* d = reinterpret_cast<uint4*>(sb);
#pragma unroll 4
    for (int w = threadIdx.x; w < 9 * NT * 8 * ks / 8; w += WARPS * 32) d[w] = src[w];
  }
  __syncthreads();
  float acc[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[nt][q] = 0.f;
  for (int ti = 0; ti < 3; ++ti) {
    const int row = sgn > 0 ? ti : 2 - ti, ii = i + (row - 1) * dil;
    if (ii < 0 || ii >= nrg) continue;        // the same for the whole CTA
    for (int tj = 0; tj < 3; ++tj) {
      const __nv_bfloat16* bt = sb + (ti * 3 + tj) * NT * 8 * ks;
      const __nv_bfloat16* xa =
          sx + ((int64_t)row * ncol + (sgn > 0 ? tj : 2 - tj) * step + 16 * warp + (lane & 15)) * ks + (lane >> 4) * 8;
      for (int k0 = 0; k0 < kpad; k0 += 16) {
        uint32_t a[4];
        ldsm_x4(a, xa + k0);
        if (NT == 1) {
          uint32_t b0, b1;
          ldsm_x2(b0, b1, bt + (lane & 7) * ks + k0 + ((lane >> 3) & 1) * 8);
          mma_bf16_16816(acc[0], a, b0, b1);
        } else {
#pragma unroll
          for (int np = 0; np < NT / 2; ++np) {
            uint32_t r[4];
            ldsm_x4(r, bt + ((2 * np + (lane >> 4)) * 8 + (lane & 7)) * ks + k0 + ((lane >> 3) & 1) * 8);
            mma_bf16_16816(acc[2 * np], a, r[0], r[1]);
            mma_bf16_16816(acc[2 * np + 1], a, r[2], r[3]);
          }
        }
      }
    }
  }
  // result to [column][point] in shared memory (over the window), out in 16-byte rows
  __syncthreads();
  float* so = reinterpret_cast<float*>(sx);
  {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        so[(nt * 8 + 2 * t + (q & 1)) * OS + 16 * warp + g + ((q & 2) ? 8 : 0)] = acc[nt][q];
  }
  __syncthreads();
  constexpr int kLr = TJ / 4;                 // lanes per row of the tile
#pragma unroll
  for (int e = threadIdx.x; e < NT * 8 * kLr; e += WARPS * 32) {
    const int n = e / kLr, p = 4 * (e - n * kLr);
    if (n >= nch || j0 + p >= ntg) continue;
    const float4 r = *reinterpret_cast<const float4*>(so + n * OS + p);
    const int64_t o = (int64_t)b * nch * plane + (int64_t)n * plane + (int64_t)i * ntg + j0 + p;
    const float bn = bias ? bias[n] : 0.f;
    float v[4] = {r.x + bn, r.y + bn, r.z + bn, r.w + bn};
    if (relu) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (v[q] < 0.f) v[q] = 0.f;
    }
    if (mask) {
      const float4 m = *reinterpret_cast<const float4*>(mask + o);
      if (!(m.x > 0.f)) v[0] = 0.f;
      if (!(m.y > 0.f)) v[1] = 0.f;
      if (!(m.z > 0.f)) v[2] = 0.f;
      if (!(m.w > 0.f)) v[3] = 0.f;
    }
    if (affine) {
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = __fadd_rn(__fmul_rn(v[q], scale), shift);
    }
    *reinterpret_cast<float4*>(Y + o) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// dX[b][ci][i][j] = sum_co sum_taps W[co][ci][tap] dY[b][co][i-(ti-1)d][j-(tj-1)d]
// (zero where mask <= 0: the gradient through the ReLU of the layer below)
template <int CIN>
__global__ void __launch_bounds__(256) k_conv_bwd_data(const float* __restrict__ dY, const float* __restrict__ W,
                                                       const float* __restrict__ mask, float* __restrict__ dX, int cout,
                                                       int nrg, int ntg, int dil) {
  extern __shared__ float sw[];  // cout * CIN * 9
  const int nw = cout * CIN * 9;
  for (int k = threadIdx.x; k < nw; k += blockDim.x) sw[k] = W[k];
  __syncthreads();
  const int b = blockIdx.z, i = blockIdx.y;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= ntg) return;
  float acc[CIN];
#pragma unroll
  for (int ci = 0; ci < CIN; ++ci) acc[ci] = 0.f;
  const int64_t plane = (int64_t)nrg * ntg;
  for (int co = 0; co < cout; ++co) {
    const float* Dc = dY + ((int64_t)b * cout + co) * plane;
#pragma unroll
    for (int ti = 0; ti < 3; ++ti) {
      const int ii = i - (ti - 1) * dil;
      if (ii < 0 || ii >= nrg) continue;
#pragma unroll
      for (int tj = 0; tj < 3; ++tj) {
        int jj = j - (tj - 1) * dil;
        jj = ((jj % ntg) + ntg) % ntg;
        const float dv = Dc[(int64_t)ii * ntg + jj];
#pragma unroll
        for (int ci = 0; ci < CIN; ++ci) acc[ci] += sw[(co * CIN + ci) * 9 + ti * 3 + tj] * dv;
      }
    }
  }
#pragma unroll
  for (int ci = 0; ci < CIN; ++ci) {
    const int64_t o = ((int64_t)b * CIN + ci) * plane + (int64_t)i * ntg + j;
    dX[o] = mask[o] > 0.f ? acc[ci] : 0.f;
  }
}

// Weight gradient: dW[co][ci][tap] = sum over batch and grid points of
// dY[b][co][p] X[b][ci][p + tap], db[co] = sum dY: a GEMM of cout x 9 cin whose
// long dimension is the grid, in FP32 FMA.  A CTA walks over row windows of 64
// points: X (three rows) and dY of a window are staged in shared memory with
// the channels consecutive, a lane owns one input channel (cin < 32: and one of
// 32 / cin points), a warp 8 output channels, so a thread keeps 8 x 9 sums in
// registers and every point costs it 9 + 2 shared loads for 72 FMA (with fewer
// output channels the warps share the points).  The CTA's sums go to a
// workspace that k_conv_bwd_w_sum adds up in a fixed order (in FP64), so the
// result does not depend on scheduling.
// Bound by FP32 FMA (2.4 G per 32 -> 32 layer at 65 x 512, batch 8).  The form
// it replaces, one CTA per (co, ci) re-reading both arrays from L2, took
// 3.4-3.9 ms for such a layer.
constexpr int kBwTj = 64;
constexpr int kBwCtas = 444;   // 3 per SM
template <int CIN, int COUT>
struct BwTile {
  static constexpr int kCot = COUT < 8 ? COUT : 8;     // output channels per thread
  static constexpr int kGroups = COUT / kCot;          // warps that differ in output channels
  static constexpr int kShare = 4 / kGroups;           // warps that share the points
  static constexpr int kPts = 32 / CIN;                // points per warp step
  static constexpr int kXs = CIN + 1, kGs = COUT < 4 ? COUT : COUT + 4;
  static constexpr int kSet = COUT * CIN * 9 + COUT;   // one set of sums
  static size_t smem(int dil) { return sizeof(float) * (kBwTj * kGs + 3 * (size_t)win_cols(kBwTj, dil) * kXs); }
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(128) k_conv_bwd_w(const float* __restrict__ X, const float* __restrict__ dY,
                                                    float* __restrict__ part, int nb, int nrg, int ntg, int dil) {
  typedef BwTile<CIN, COUT> T;
  extern __shared__ __align__(16) float bw_raw[];
  float* sg = bw_raw;                                  // [point][co]
  float* sx = bw_raw + kBwTj * T::kGs;                 // [row][column][ci]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int cog = w % T::kGroups, wj = w / T::kGroups, ci = lane % CIN, ps = lane / CIN;
  const int ncol = win_cols(kBwTj, dil), step = dil < kBwTj ? dil : kBwTj;
  const int nwin = (ntg + kBwTj - 1) / kBwTj;
  const int64_t plane = (int64_t)nrg * ntg;
  LanePoints<kBwTj> pts;
  float acc[T::kCot][9], bsum[(COUT + 3) / 4];
#pragma unroll
  for (int c = 0; c < T::kCot; ++c)
#pragma unroll
    for (int k = 0; k < 9; ++k) acc[c][k] = 0.f;
#pragma unroll
  for (int q = 0; q < (COUT + 3) / 4; ++q) bsum[q] = 0.f;
  for (int64_t u = blockIdx.x; u < (int64_t)nb * nrg * nwin; u += gridDim.x) {
    const int win = (int)(u % nwin);
    const int64_t bi = u / nwin;
    const int i = (int)(bi % nrg), b = (int)(bi / nrg), j0 = win * kBwTj;
#pragma unroll
    for (int q = 0; q < (COUT + 3) / 4; ++q) {
      const int co = w + 4 * q;
      if (co < COUT) {
        const float* src = dY + ((int64_t)b * COUT + co) * plane + (int64_t)i * ntg;
#pragma unroll
        for (int p = lane; p < kBwTj; p += 32) {
          const float v = j0 + p < ntg ? src[j0 + p] : 0.f;
          sg[p * T::kGs + co] = v;
          bsum[q] += v;
        }
      }
    }
    pts.set(lane, ncol, j0, dil, ntg);
#pragma unroll 1
    for (int row = 0; row < 3; ++row) {
      const int ii = i + (row - 1) * dil;
      const bool in = ii >= 0 && ii < nrg;
      const float* src = X + (int64_t)b * CIN * plane + (int64_t)(in ? ii : 0) * ntg;
#pragma unroll
      for (int k = 0; k < LanePoints<kBwTj>::kMax; ++k) {
        if (pts.j[k] < 0) continue;
        float* dst = sx + (row * ncol + lane + 32 * k) * T::kXs;
        float v[(CIN + 3) / 4];
#pragma unroll
        for (int q = 0; q < CIN / 4; ++q) v[q] = in ? src[(int64_t)(w + 4 * q) * plane + pts.j[k]] : 0.f;
#pragma unroll
        for (int q = 0; q < CIN / 4; ++q) dst[w + 4 * q] = v[q];
      }
    }
    __syncthreads();
#pragma unroll 2
    for (int pp = wj; pp < kBwTj / T::kPts; pp += T::kShare) {
      const int p = pp * T::kPts + ps;
      float g[T::kCot], x[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) x[k] = sx[((k / 3) * ncol + p + (k % 3) * step) * T::kXs + ci];
      if (T::kCot == 8) {
        const float4 u0 = *reinterpret_cast<const float4*>(sg + p * T::kGs + 8 * cog);
        const float4 u1 = *reinterpret_cast<const float4*>(sg + p * T::kGs + 8 * cog + 4);
        const float gg[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
        for (int c = 0; c < T::kCot; ++c) g[c] = gg[c];
      } else {
#pragma unroll
        for (int c = 0; c < T::kCot; ++c) g[c] = sg[p * T::kGs + c];
      }
#pragma unroll
      for (int c = 0; c < T::kCot; ++c)
#pragma unroll
        for (int k = 0; k < 9; ++k) acc[c][k] += g[c] * x[k];
    }
    __syncthreads();
  }
  float* out = part + ((int64_t)blockIdx.x * T::kShare + wj) * T::kSet;
#pragma unroll
  for (int c = 0; c < T::kCot; ++c) {
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      float v = acc[c][k];
#pragma unroll
      for (int o = CIN; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (ps == 0) out[((cog * T::kCot + c) * CIN + ci) * 9 + k] = v;
    }
  }
  float* ob = part + (int64_t)blockIdx.x * T::kShare * T::kSet + COUT * CIN * 9;   // bias: the CTA's first set
#pragma unroll
  for (int q = 0; q < (COUT + 3) / 4; ++q) {
    float v = bsum[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0 && w + 4 * q < COUT) ob[w + 4 * q] = v;
  }
}

// grad[e] = sum over the CTAs' sets (the bias, e >= nw, over the first set of each
// CTA), 32 values x 32 parts of the sets per CTA
__global__ void __launch_bounds__(1024) k_conv_bwd_w_sum(const float* __restrict__ part, float* __restrict__ dW,
                                                         float* __restrict__ db, int nw, int nset_len, int nsets,
                                                         int share) {
  const int e = blockIdx.x * 32 + (threadIdx.x & 31), y = threadIdx.x >> 5;
  double s = 0.0;
  if (e < nset_len) {
    const int stride = e < nw ? 1 : share;
#pragma unroll 8
    for (int k = y * stride; k < nsets; k += 32 * stride) s += (double)part[(int64_t)k * nset_len + e];
  }
  __shared__ double sh[32][33];
  sh[y][threadIdx.x & 31] = s;
  __syncthreads();
  s = sh[threadIdx.x & 31][y];   // warp y: the 32 parts of value y
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  const int ey = blockIdx.x * 32 + y;
  if ((threadIdx.x & 31) == 0 && ey < nset_len) {
    if (ey < nw) dW[ey] = (float)s;
    else db[ey - nw] = (float)s;
  }
}

// MSE loss L = mean (y - t)^2 and dL/dy
__global__ void __launch_bounds__(kRedThreads) k_mse(const float* __restrict__ y, const float* __restrict__ t,
                                                     float* __restrict__ g, int64_t n, double* partial,
                                                     unsigned int* counter, double* out) {
  double s = 0.0;
  const float inv = 2.0f / (float)n;
  for (int64_t i = blockIdx.x * (int64_t)kRedThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kRedThreads) {
    const float d = y[i] - t[i];
    g[i] = inv * d;
    s += (double)d * (double)d;
  }
  double v[1] = {s / (double)n};
  double* o[1] = {out};
  grid_finish<1>(v, partial, counter, o);
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       int64_t n, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// ---- host: layer dispatch ----------------------------------------------------------
template <int N>
static void conv_fwd_n(Cnn& n, cudaStream_t s, int l, const float* X, float* Y, int nb) {
  const int cin = n.cin_of(l);
  const size_t smem = sizeof(float) * (N * cin * 9 + N);
  dim3 grid((unsigned)div_up(n.ntg, 256), (unsigned)n.nrg, (unsigned)nb);
  ++g_klaunch;
  k_conv_fwd<N><<<grid, 256, smem, s>>>(X, n.param + n.woff[l], n.param + n.boff[l], Y, cin, n.nrg, n.ntg,
                                                 n.dil[l], l < n.L - 1 ? 1 : 0);
}
static void conv_fwd(Cnn& n, cudaStream_t s, int l, const float* X, float* Y, int nb) {
  switch (n.cout_of(l)) {
    case 1: conv_fwd_n<1>(n, s, l, X, Y, nb); break;
    case 8: conv_fwd_n<8>(n, s, l, X, Y, nb); break;
    case 16: conv_fwd_n<16>(n, s, l, X, Y, nb); break;
    case 32: conv_fwd_n<32>(n, s, l, X, Y, nb); break;
    default: throw std::runtime_error("unsupported channel count");
  }
  DP_LAUNCH_CHECK();
}
template <int N>
static void conv_bwd_data_n(Cnn& n, int l, const float* dY, const float* mask, float* dX, int nb) {
  const int cout = n.cout_of(l);
  const size_t smem = sizeof(float) * (cout * N * 9);
  dim3 grid((unsigned)div_up(n.ntg, 256), (unsigned)n.nrg, (unsigned)nb);
  ++g_klaunch;
  k_conv_bwd_data<N><<<grid, 256, smem, n.stream>>>(dY, n.param + n.woff[l], mask, dX, cout, n.nrg, n.ntg,
                                                     n.dil[l]);
}
static void conv_bwd_data(Cnn& n, int l, const float* dY, const float* mask, float* dX, int nb) {
  switch (n.cin_of(l)) {
    case 4: conv_bwd_data_n<4>(n, l, dY, mask, dX, nb); break;
    case 8: conv_bwd_data_n<8>(n, l, dY, mask, dX, nb); break;
    case 16: conv_bwd_data_n<16>(n, l, dY, mask, dX, nb); break;
    case 32: conv_bwd_data_n<32>(n, l, dY, mask, dX, nb); break;
    default: throw std::runtime_error("unsupported channel count");
  }
  DP_LAUNCH_CHECK();
}

// ---- tensor-core dispatch ------------------------------------------------------------
static int pad16(int c) { return (c + 15) / 16 * 16; }
static int ntiles(int c) { return (c + 7) / 8; }
// elements of a layer's B operand: forward (n = cout, k = cin) or data gradient (n = cin, k = cout)
static int64_t wk_elems(int cin, int cout, bool transpose) {
  const int nch = transpose ? cin : cout, kch = transpose ? cout : cin;
  return 9LL * ntiles(nch) * 8 * (pad16(kch) + 8);
}
static bool tc_ok(const Cnn& n) { return n.bf16 && n.ntg % 16 == 0; }

// 128-point tiles where the grid then still has 4 CTAs per SM, else 64-point
// ones (65 x 512, batch 1: 260 or 520 CTAs).  Y and mask rows are read and
// written in 16-byte groups: a caller's y that is not 16-byte aligned is staged
// by the caller of this (see cnn_forward).
template <int NT, int WARPS>
static void conv_tc_nw(Cnn& n, cudaStream_t s, const float* X, const __nv_bfloat16* Bk, const float* bias,
                       const float* mask, float* Y, int kch, int nch, int dil, int sgn, int relu, int nb, int affine,
                       float scale, float shift) {
  const int kpad = pad16(kch);
  const size_t smem = ConvTile<NT, WARPS>::smem(kpad, dil);
  if (smem > 48 * 1024)
    DP_CUDA(cudaFuncSetAttribute(k_conv_tc<NT, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  dim3 grid((unsigned)div_up(n.ntg, ConvTile<NT, WARPS>::kTj), (unsigned)n.nrg, (unsigned)nb);
  ++g_klaunch;
  k_conv_tc<NT, WARPS><<<grid, WARPS * 32, smem, s>>>(X, Bk, bias, mask, Y, kch, kpad, nch, n.nrg, n.ntg, dil, sgn,
                                                      relu, affine, scale, shift);
  DP_LAUNCH_CHECK();
}
template <int NT>
static void conv_tc_n(Cnn& n, cudaStream_t s, const float* X, const __nv_bfloat16* Bk, const float* bias,
                      const float* mask, float* Y, int kch, int nch, int dil, int sgn, int relu, int nb, int affine,
                      float scale, float shift) {
  if (div_up(n.ntg, 128) * n.nrg * nb >= 4 * 148)
    conv_tc_nw<NT, 8>(n, s, X, Bk, bias, mask, Y, kch, nch, dil, sgn, relu, nb, affine, scale, shift);
  else
    conv_tc_nw<NT, 4>(n, s, X, Bk, bias, mask, Y, kch, nch, dil, sgn, relu, nb, affine, scale, shift);
}
static void conv_tc(Cnn& n, cudaStream_t s, const float* X, const __nv_bfloat16* Bk, const float* bias,
                    const float* mask, float* Y, int kch, int nch, int dil, int sgn, int relu, int nb, int affine = 0,
                    float scale = 1.f, float shift = 0.f) {
  switch (ntiles(nch)) {
    case 1: conv_tc_n<1>(n, s, X, Bk, bias, mask, Y, kch, nch, dil, sgn, relu, nb, affine, scale, shift); break;
    case 2: conv_tc_n<2>(n, s, X, Bk, bias, mask, Y, kch, nch, dil, sgn, relu, nb, affine, scale, shift); break;
    case 4: conv_tc_n<4>(n, s, X, Bk, bias, mask, Y, kch, nch, dil, sgn, relu, nb, affine, scale, shift); break;
    default: throw std::runtime_error("unsupported channel count");
  }
}
// the BF16 operands of the current weights (after every change of the weights)
static void refresh_weights(Cnn& n, cudaStream_t s) {
  WkArgs a{};
  for (int l = 0; l < n.L; ++l) {
    a.w[l] = n.woff[l];
    a.o[2 * l] = n.wkoff[2 * l];
    a.o[2 * l + 1] = n.wkoff[2 * l + 1];
    a.cin[l] = n.cin_of(l);
    a.cout[l] = n.cout_of(l);
  }
  ++g_klaunch;
  k_conv_weights_bf16<<<dim3(16, 2 * n.L), 256, 0, s>>>(n.param, n.wk, a);
  DP_LAUNCH_CHECK();
}

// CTAs of a weight gradient, and the floats of a layer's partial sums: kShare sets
// (BwTile) for each
static int bw_ctas(const Cnn& n, int nb) {
  return (int)std::min<int64_t>(kBwCtas, (int64_t)nb * n.nrg * div_up(n.ntg, kBwTj));
}
static int64_t bw_part_floats(const Cnn& n, int l) {
  const int cin = n.cin_of(l), cout = n.cout_of(l), groups = cout / std::min(cout, 8);
  return (int64_t)bw_ctas(n, n.bmax) * (4 / groups) * (cout * cin * 9 + cout);
}
static_assert(BwTile<8, 16>::kShare == 2 && BwTile<4, 1>::kShare == 4 && BwTile<32, 32>::kShare == 1 &&
              BwTile<8, 16>::kSet == 16 * 8 * 9 + 16, "bw_part_floats follows BwTile");

template <int CIN, int COUT>
static void conv_bwd_w_t(Cnn& n, int l, const float* X, const float* dY, int nb) {
  typedef BwTile<CIN, COUT> T;
  const size_t smem = T::smem(n.dil[l]);
  if (smem > 48 * 1024)
    DP_CUDA(cudaFuncSetAttribute(k_conv_bwd_w<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int ctas = bw_ctas(n, nb);
  ++g_klaunch;
  k_conv_bwd_w<CIN, COUT><<<ctas, 128, smem, n.stream>>>(X, dY, n.wpart, nb, n.nrg, n.ntg, n.dil[l]);
  ++g_klaunch;
  k_conv_bwd_w_sum<<<(int)div_up(T::kSet, 32), 1024, 0, n.stream>>>(n.wpart, n.grad + n.woff[l], n.grad + n.boff[l],
                                                                   COUT * CIN * 9, T::kSet, ctas * T::kShare,
                                                                   T::kShare);
  DP_LAUNCH_CHECK();
}
template <int CIN>
static void conv_bwd_w_n(Cnn& n, int l, const float* X, const float* dY, int nb) {
  switch (n.cout_of(l)) {
    case 1: conv_bwd_w_t<CIN, 1>(n, l, X, dY, nb); break;
    case 8: conv_bwd_w_t<CIN, 8>(n, l, X, dY, nb); break;
    case 16: conv_bwd_w_t<CIN, 16>(n, l, X, dY, nb); break;
    case 32: conv_bwd_w_t<CIN, 32>(n, l, X, dY, nb); break;
    default: throw std::runtime_error("unsupported channel count");
  }
}
static void conv_bwd_w(Cnn& n, int l, const float* X, const float* dY, int nb) {
  switch (n.cin_of(l)) {
    case 4: conv_bwd_w_n<4>(n, l, X, dY, nb); break;
    case 8: conv_bwd_w_n<8>(n, l, X, dY, nb); break;
    case 16: conv_bwd_w_n<16>(n, l, X, dY, nb); break;
    case 32: conv_bwd_w_n<32>(n, l, X, dY, nb); break;
    default: throw std::runtime_error("unsupported channel count");
  }
}

__global__ void k_affine(float* __restrict__ y, int64_t n, float scale, float shift) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = __fadd_rn(__fmul_rn(y[i], scale), shift);
}

// x -> y (null: the network's own output buffer); affine: y * scale + shift
static void cnn_forward(Cnn& n, cudaStream_t s, const float* x, float* y, int nb, int affine = 0, float scale = 1.f,
                        float shift = 0.f) {
  n.act[0] = const_cast<float*>(x);
  for (int l = 0; l < n.L; ++l) {
    const bool last = l == n.L - 1;
    // straight into the caller's y where the kernel's 16-byte stores can reach it
    float* out = last && y && in_place(n.device, y, DP_MEM_DEVICE, 16) ? y : n.act[l + 1];
    if (tc_ok(n)) {
      conv_tc(n, s, n.act[l], n.wk + n.wkoff[2 * l], n.param + n.boff[l], nullptr, out, n.cin_of(l), n.cout_of(l),
              n.dil[l], 1, last ? 0 : 1, nb, last ? affine : 0, scale, shift);
    } else {
      conv_fwd(n, s, l, n.act[l], out, nb);
      if (last && affine) {
        const int64_t m = (int64_t)nb * n.nrg * n.ntg;
        ++g_klaunch;
        k_affine<<<(int)div_up(m, 256), 256, 0, s>>>(out, m, scale, shift);
        DP_LAUNCH_CHECK();
      }
    }
    if (last && y && out != y)
      DP_CUDA(cudaMemcpyAsync(y, out, sizeof(float) * nb * (int64_t)n.nrg * n.ntg, cudaMemcpyDeviceToDevice, s));
  }
}

// forward + backward; returns the device loss in n.loss
static void cnn_fwd_bwd(Cnn& n, const float* x, const float* t, int nb) {
  cnn_forward(n, n.stream, x, nullptr, nb);
  const int64_t plane = (int64_t)n.nrg * n.ntg;
  const int64_t nout = (int64_t)nb * plane;
  float* g = n.dbuf0;
  float* g2 = n.dbuf1;
  ++g_klaunch;
  k_mse<<<red_grid(nout), kRedThreads, 0, n.stream>>>(n.act[n.L], t, g, nout, n.partial, n.counter, n.loss);
  DP_LAUNCH_CHECK();
  for (int l = n.L - 1; l >= 0; --l) {
    const int cin = n.cin_of(l), cout = n.cout_of(l);
    conv_bwd_w(n, l, n.act[l], g, nb);
    if (l > 0) {
      // the data gradient leaves through the ReLU of layer l - 1 (zero where its output is)
      if (tc_ok(n))
        conv_tc(n, n.stream, g, n.wk + n.wkoff[2 * l + 1], nullptr, n.act[l], g2, cout, cin, n.dil[l], -1, 0, nb);
      else
        conv_bwd_data(n, l, g, n.act[l], g2, nb);
      std::swap(g, g2);
    }
  }
}

// ---- input features and the prolongation of the predicted pressure -----------------
// grid point (i, j) = fine vertex (2i, 2j) = lattice node (4i, 4j); features from the
// element of type 0 in fine cell (min(2i, ncr-1), 2j)
// (normalised: (v - mean) / std per channel, in FP32)
struct CnnNorm {
  float mean[4], std[4];
  int on;
};
__global__ void k_cnn_inputs(const double* __restrict__ rho_lat, const double* __restrict__ eta,
                             const double* __restrict__ C, int mat_kind, int nel, int ncr, int nct, int A,
                             float* __restrict__ X, int nrg, int ntg, CnnNorm nm) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (j >= ntg) return;
  const int a = 4 * i, b = 4 * j;
  const int ir = min(2 * i, ncr - 1), it = 2 * j;
  const int e = 2 * (ir + ncr * it);
  double le = 0.0;
  for (int ip = 0; ip < 6; ++ip) le += log10(eta[(size_t)ip * nel + e]);
  double c2 = 1.0, s2 = 0.0;
  if (mat_kind == MAT_TI) {
    const double dx = C[nel + e], dy = C[2 * (size_t)nel + e];
    const double nn = dx * dx + dy * dy;
    if (nn > 0) { c2 = (dx * dx - dy * dy) / nn; s2 = 2.0 * dx * dy / nn; }
  }
  const int64_t plane = (int64_t)nrg * ntg, off = (int64_t)i * ntg + j;
  const float v[4] = {(float)rho_lat[a + (int64_t)A * b], (float)(le / 6.0), (float)c2, (float)s2};
#pragma unroll
  for (int k = 0; k < 4; ++k)
    X[k * plane + off] = nm.on ? __fdiv_rn(__fsub_rn(v[k], nm.mean[k]), nm.std[k]) : v[k];
}

// bilinear value of the grid field at fine vertex (ir, it) = grid (ir/2, it/2)
__device__ inline double grid_at(const float* p, int ir, int it, int nrg, int ntg) {
  const int i0 = ir >> 1, j0 = it >> 1;
  const int i1 = (ir & 1) ? min(i0 + 1, nrg - 1) : i0;
  const int j1 = (it & 1) ? (j0 + 1 == ntg ? 0 : j0 + 1) : j0;
  return 0.25 * ((double)p[(int64_t)i0 * ntg + j0] + (double)p[(int64_t)i1 * ntg + j0] +
                 (double)p[(int64_t)i0 * ntg + j1] + (double)p[(int64_t)i1 * ntg + j1]);
}

__global__ void k_guess_prolong(const float* __restrict__ pg, int nrg, int ntg, double scale, int ncr, int nct,
                                int pressure, double* __restrict__ P, int nel) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nel) return;
  const int q = e >> 1, t = e & 1;
  const int ir = q % ncr, it = q / ncr;
  const int it1 = it + 1 == nct ? 0 : it + 1;
  int vr[3], vt[3];
  if (t == 0) { vr[0] = ir; vt[0] = it; vr[1] = ir; vt[1] = it1; vr[2] = ir + 1; vt[2] = it; }
  else { vr[0] = ir; vt[0] = it1; vr[1] = ir + 1; vt[1] = it1; vr[2] = ir + 1; vt[2] = it; }
  for (int k = 0; k < 3; ++k) {
    const double v = scale * grid_at(pg, vr[k], vt[k], nrg, ntg);
    if (pressure == 1) P[3 * (int64_t)e + k] = v;
    else P[vr[k] + (int64_t)(ncr + 1) * vt[k]] = v;  // shared vertices get identical values
  }
}

}  // namespace dp

struct dp_cnn {
  dp::Cnn n;
};

using namespace dp;

extern "C" {

int dp_cnn_create(int32_t nrg, int32_t ntg, int32_t channels, int32_t layers, const int32_t* dilations,
                  int32_t max_batch, int32_t device, dp_cnn** out) {
  if (!out) return DP_BAD_ARG;
  *out = nullptr;
  dp_cnn* h = nullptr;
  int st = guarded(nullptr, [&] {
    if (nrg < 2 || ntg < 3 || layers < 2 || layers > kCnnMaxLayers || max_batch < 1)
      throw BadArg("invalid network shape");
    if (channels != 8 && channels != 16 && channels != 32) throw BadArg("channels must be 8, 16 or 32");
    h = new dp_cnn();
    Cnn& n = h->n;
    n.nrg = nrg; n.ntg = ntg; n.C = channels; n.L = layers; n.device = device; n.bmax = max_batch;
    for (int l = 0; l < layers; ++l) {
      n.dil[l] = dilations ? dilations[l] : 1;
      if (n.dil[l] < 1 || n.dil[l] >= nrg) throw BadArg("invalid dilation");
    }
    DP_CUDA(cudaSetDevice(device));
    DP_CUDA(cudaStreamCreateWithFlags(&n.stream, cudaStreamNonBlocking));
    int64_t off = 0;
    for (int l = 0; l < layers; ++l) {
      n.woff.push_back(off);
      off += (int64_t)n.cout_of(l) * n.cin_of(l) * 9;
      n.boff.push_back(off);
      off += n.cout_of(l);
    }
    n.nparam = off;
    DP_CUDA(cudaMalloc(&n.param, sizeof(float) * off));
    DP_CUDA(cudaMalloc(&n.grad, sizeof(float) * off));
    DP_CUDA(cudaMalloc(&n.adam_m, sizeof(float) * off));
    DP_CUDA(cudaMalloc(&n.adam_v, sizeof(float) * off));
    // zeroed on the network's own stream, which dp_cnn_set_params writes them on and
    // which does not wait for the default stream
    DP_CUDA(cudaMemsetAsync(n.param, 0, sizeof(float) * off, n.stream));
    DP_CUDA(cudaMemsetAsync(n.adam_m, 0, sizeof(float) * off, n.stream));
    DP_CUDA(cudaMemsetAsync(n.adam_v, 0, sizeof(float) * off, n.stream));
    const int64_t plane = (int64_t)nrg * ntg;
    n.act.assign(layers + 1, nullptr);
    for (int l = 0; l < layers; ++l) DP_CUDA(cudaMalloc(&n.act[l + 1], sizeof(float) * max_batch * n.cout_of(l) * plane));
    // both gradient buffers and the weight gradient's workspace: an allocation costs
    // ~0.35 ms whatever its size
    const int64_t gmax = div_up((int64_t)max_batch * std::max(channels, 4) * plane, 64) * 64;   // 256-byte steps
    int64_t part = 0;
    for (int l = 0; l < layers; ++l) part = std::max(part, bw_part_floats(n, l));
    DP_CUDA(cudaMalloc(&n.dbuf0, sizeof(float) * (2 * gmax + part)));
    n.dbuf1 = n.dbuf0 + gmax;
    n.wpart = n.dbuf1 + gmax;
    int64_t wtot = 0;
    for (int k = 0; k < 2 * layers; ++k) {
      n.wkoff.push_back(wtot);
      wtot += wk_elems(n.cin_of(k / 2), n.cout_of(k / 2), k & 1);   // a multiple of 8 elements: 16-byte aligned
    }
    DP_CUDA(cudaMalloc(&n.wk, sizeof(__nv_bfloat16) * wtot));
    DP_CUDA(cudaMemsetAsync(n.wk, 0, sizeof(__nv_bfloat16) * wtot, n.stream));   // the operands of zero weights
    DP_CUDA(cudaMalloc(&n.partial, sizeof(double) * 4 * kRedBlocks));
    DP_CUDA(cudaMalloc(&n.counter, sizeof(unsigned int)));
    DP_CUDA(cudaMemsetAsync(n.counter, 0, sizeof(unsigned int), n.stream));
    DP_CUDA(cudaMalloc(&n.loss, sizeof(double)));
    DP_CUDA(cudaMallocHost(&n.h_loss, sizeof(double)));
    DP_CUDA(cudaStreamSynchronize(n.stream));   // dp_guess_predict reads the weights on the context's stream
    return (int)DP_OK;
  });
  if (st != DP_OK) {
    delete h;
    return st;
  }
  *out = h;
  return DP_OK;
}

void dp_cnn_destroy(dp_cnn* h) {
  if (!h) return;
  cudaSetDevice(h->n.device);
  if (h->n.stream) cudaStreamSynchronize(h->n.stream);
  delete h;
}

int64_t dp_cnn_num_params(const dp_cnn* h) { return h ? h->n.nparam : -1; }

int dp_cnn_set_math(dp_cnn* h, int32_t bf16) {
  if (!h || bf16 < 0 || bf16 > 1) return DP_BAD_ARG;
  h->n.bf16 = bf16;
  return DP_OK;
}

int dp_cnn_set_params(dp_cnn* h, const float* p, int64_t n) {
  if (!h || !p || n != h->n.nparam) return DP_BAD_ARG;
  return guarded(nullptr, [&] {
    DP_CUDA(cudaSetDevice(h->n.device));
    cudaStream_t s = h->n.stream;
    DP_CUDA(cudaMemcpyAsync(h->n.param, p, sizeof(float) * n, cudaMemcpyHostToDevice, s));
    DP_CUDA(cudaMemsetAsync(h->n.adam_m, 0, sizeof(float) * n, s));
    DP_CUDA(cudaMemsetAsync(h->n.adam_v, 0, sizeof(float) * n, s));
    refresh_weights(h->n, s);
    DP_CUDA(cudaStreamSynchronize(s));
    h->n.step = 0;
    return (int)DP_OK;
  });
}

int dp_cnn_get_params(dp_cnn* h, float* p, float* g, int64_t n) {
  if (!h || n != h->n.nparam) return DP_BAD_ARG;
  return guarded(nullptr, [&] {
    DP_CUDA(cudaSetDevice(h->n.device));
    if (p) DP_CUDA(cudaMemcpy(p, h->n.param, sizeof(float) * n, cudaMemcpyDeviceToHost));
    if (g) DP_CUDA(cudaMemcpy(g, h->n.grad, sizeof(float) * n, cudaMemcpyDeviceToHost));
    return (int)DP_OK;
  });
}

int dp_cnn_forward(dp_cnn* h, const float* x, float* y, int32_t nb) {
  if (!h || !x || !y || nb < 1 || nb > h->n.bmax) return DP_BAD_ARG;
  return guarded(nullptr, [&] {
    Cnn& n = h->n;
    DP_CUDA(cudaSetDevice(n.device));
    cnn_forward(n, n.stream, x, y, nb);
    DP_CUDA(cudaStreamSynchronize(n.stream));
    return (int)DP_OK;
  });
}

int dp_cnn_gradients(dp_cnn* h, const float* x, const float* t, int32_t nb, double* loss) {
  if (!h || !x || !t || nb < 1 || nb > h->n.bmax) return DP_BAD_ARG;
  return guarded(nullptr, [&] {
    Cnn& n = h->n;
    DP_CUDA(cudaSetDevice(n.device));
    cnn_fwd_bwd(n, x, t, nb);
    DP_CUDA(cudaMemcpyAsync(n.h_loss, n.loss, sizeof(double), cudaMemcpyDeviceToHost, n.stream));
    DP_CUDA(cudaStreamSynchronize(n.stream));
    if (loss) *loss = *n.h_loss;
    return (int)DP_OK;
  });
}

int dp_cnn_train_step(dp_cnn* h, const float* x, const float* t, int32_t nb, float lr, double* loss) {
  if (!h || !x || !t || nb < 1 || nb > h->n.bmax || !(lr > 0.f)) return DP_BAD_ARG;
  return guarded(nullptr, [&] {
    Cnn& n = h->n;
    DP_CUDA(cudaSetDevice(n.device));
    cnn_fwd_bwd(n, x, t, nb);
    n.step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)n.step), c2 = 1.f - std::pow(b2, (float)n.step);
    ++g_klaunch;
    k_adam<<<(int)div_up(n.nparam, 256), 256, 0, n.stream>>>(n.param, n.grad, n.adam_m, n.adam_v, n.nparam, lr, b1,
                                                               b2, 1e-8f, c1, c2);
    DP_LAUNCH_CHECK();
    refresh_weights(n, n.stream);
    DP_CUDA(cudaMemcpyAsync(n.h_loss, n.loss, sizeof(double), cudaMemcpyDeviceToHost, n.stream));
    DP_CUDA(cudaStreamSynchronize(n.stream));
    if (loss) *loss = *n.h_loss;
    return (int)DP_OK;
  });
}

static void launch_cnn_inputs(Ctx& c, float* x, int nrg, int ntg, const CnnNorm& nm) {
  if (c.fine.ncr % 2 || c.fine.nct % 2) throw BadArg("the guess grid needs even cell counts");
  if (nrg != c.fine.ncr / 2 + 1 || ntg != c.fine.nct / 2) throw BadArg("grid must be (ncr/2+1) x (nct/2)");
  if (c.mat_kind == MAT_NONE) throw BadArg("material not set");
  dim3 grid((unsigned)div_up(ntg, 128), (unsigned)nrg);
  ++g_klaunch;
  k_cnn_inputs<<<grid, 128, 0, c.stream>>>(c.rho_lat, c.eta, c.C, c.mat_kind, (int)c.fine.nel, c.fine.ncr, c.fine.nct,
                                           (int)c.fine.A(), x, nrg, ntg, nm);
  DP_LAUNCH_CHECK();
}

// scale * grid field -> pressure DOFs in P (host or device)
static void launch_guess_prolong(Ctx& c, const float* pg, int nrg, int ntg, double scale, double* P, int mem) {
  if (nrg != c.fine.ncr / 2 + 1 || ntg != c.fine.nct / 2) throw BadArg("grid must be (ncr/2+1) x (nct/2)");
  double* dP = in_place(c.device, P, mem) ? P : (double*)c.work[W_P];
  ++g_klaunch;
  k_guess_prolong<<<(int)div_up(c.fine.nel, 256), 256, 0, c.stream>>>(pg, nrg, ntg, scale, c.fine.ncr, c.fine.nct,
                                                                      c.mesh.pressure, dP, (int)c.fine.nel);
  DP_LAUNCH_CHECK();
  if (dP != P) DP_CUDA(cudaMemcpyAsync(P, dP, sizeof(double) * c.mesh.npres, kind_out(mem), c.stream));
}

int dp_cnn_inputs(dp_ctx* h, float* x, int32_t nrg, int32_t ntg) {
  if (!h || !x) return DP_BAD_ARG;
  Ctx& c = h->c;
  return guarded(&c, [&] {
    DP_CUDA(cudaSetDevice(c.device));
    launch_cnn_inputs(c, x, nrg, ntg, CnnNorm{});
    DP_CUDA(cudaStreamSynchronize(c.stream));
    return (int)DP_OK;
  });
}

int dp_guess_from_grid(dp_ctx* h, const float* pg, int32_t nrg, int32_t ntg, double scale, double* P, int32_t mem) {
  if (!h || !pg || !P) return DP_BAD_ARG;
  Ctx& c = h->c;
  return guarded(&c, [&] {
    DP_CUDA(cudaSetDevice(c.device));
    launch_guess_prolong(c, pg, nrg, ntg, scale, P, mem);
    DP_CUDA(cudaStreamSynchronize(c.stream));
    return (int)DP_OK;
  });
}

int dp_guess_predict(dp_ctx* h, dp_cnn* net, const float* x_mean, const float* x_std, float y_mean, float y_std,
                     double scale, float* x, float* y, double* P, int32_t mem) {
  if (!h || !net || !x_mean || !x_std || !x || !y || !P) return DP_BAD_ARG;
  Ctx& c = h->c;
  return guarded(&c, [&] {
    Cnn& n = net->n;
    DP_CUDA(cudaSetDevice(c.device));
    if (n.device != c.device) throw BadArg("network and context are on different devices");
    CnnNorm nm{};
    nm.on = 1;
    for (int k = 0; k < 4; ++k) {
      nm.mean[k] = x_mean[k];
      nm.std[k] = x_std[k];
    }
    // everything on the context's stream: the network's own calls are synchronous,
    // so its buffers are free
    launch_cnn_inputs(c, x, n.nrg, n.ntg, nm);
    cnn_forward(n, c.stream, x, y, 1, 1, y_std, y_mean);
    launch_guess_prolong(c, y, n.nrg, n.ntg, scale, P, mem);
    DP_CUDA(cudaStreamSynchronize(c.stream));
    return (int)DP_OK;
  });
}

}  // extern "C"
