// VJP kernels of the implicit steady-state adjoint (reference
// steady_state_grad.py:214-233, 306-327): given lambda = J_y^{-T} v, the
// cotangents  cot = -lambda . df/dtheta  of the residual
// f = chem_rhs(y, M, k) + diffusion(y) (steady_state_grad.py:116-130) for
//   k[r, z]    (chem.py:92-125; f is linear in k),
//   M[z]       (three-body rates),
//   Kzz[m]     (eddy diffusion of the two layers sharing interface m,
//               jax_step.py:167-189),
//   top_flux, bot_flux, bot_vdep (boundary fluxes, jax_step.py:236-245).
#include <cuda_runtime.h>

#include "vb_common.cuh"
#include "vb_launch.cuh"
#include "vb_layer.cuh"

namespace vb {

constexpr int VJP_THREADS = 256;

// One CTA per (layer, atmosphere): g_k[r][z] = -P'[r] * S[r] with P' the rate
// per unit k and S = sum_s p_st lambda[p_idx] - sum_s r_st lambda[r_idx].
__global__ void __launch_bounds__(VJP_THREADS)
vjp_k_kernel(NetDev net, Batch B, const double* __restrict__ y, const double* __restrict__ k,
             const double* __restrict__ atm, double* __restrict__ ws, double* __restrict__ g_k,
             double* __restrict__ g_M) {
  __shared__ double ys[VB_MAX_NI + 1], ls[VB_MAX_NI + 1], red[VJP_THREADS / 32];
  const int b = blockIdx.y, j = blockIdx.x;
  Geo g = geo_of(B, b);
  if (j >= g.nz) return;
  const int ni = B.ni, nz = g.nz, T = net.T;
  AtmRef a = atm_ref(atm + g.atm, nz, ni);
  const double* lam = ws_view(ws, g, ni, B.ld).k1;   // lambda, [nz][ni]
  for (int i = threadIdx.x; i <= ni; i += blockDim.x) {
    ys[i] = i < ni ? y[g.z0 * ni + (int64_t)j * ni + i] : 1.0;
    ls[i] = i < ni ? lam[(int64_t)j * ni + i] : 0.0;
  }
  __syncthreads();
  const double M = a.M[j];
  const double* kc = k + g.z0 * (B.nr + 1) + j;
  double gm = 0.0;
  for (int r = threadIdx.x; r <= net.nr; r += blockDim.x) {
    double prod = 1.0, S = 0.0;
    for (int s = 0; s < T; ++s) {
      const double st = net.r_st[r * T + s];
      if (st > 0.0) prod = prod * pow_st(ys[net.r_idx[r * T + s]], st);
      S = S - st * ls[net.r_idx[r * T + s]];
      S = S + net.p_st[r * T + s] * ls[net.p_idx[r * T + s]];
    }
    const bool three = net.three[r] != 0;
    const double Pp = three ? prod * M : prod;
    if (g_k) g_k[g.z0 * (B.nr + 1) + (int64_t)r * nz + j] = -Pp * S;
    if (three) gm = gm - kc[(int64_t)r * nz] * prod * S;
  }
  if (g_M) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) gm += __shfl_xor_sync(0xffffffffu, gm, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = gm;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < VJP_THREADS / 32; ++w) t += red[w];
      g_M[g.z0 + j] = t;
    }
  }
}

// One CTA per atmosphere: eddy Kzz and boundary-flux cotangents.
__global__ void __launch_bounds__(VJP_THREADS)
vjp_transport_kernel(Batch B, const double* __restrict__ y, const double* __restrict__ atm, int flags,
                     double* __restrict__ ws, double* __restrict__ g_Kzz, double* __restrict__ g_top,
                     double* __restrict__ g_bot, double* __restrict__ g_vdep) {
  extern __shared__ double ysum[];
  const int b = blockIdx.x;
  Geo g = geo_of(B, b);
  const int ni = B.ni, nz = g.nz;
  AtmRef a = atm_ref(atm + g.atm, nz, ni);
  const double* yb = y + g.z0 * ni;
  const double* lb = ws_view(ws, g, ni, B.ld).k1;
  for (int j = threadIdx.x; j < nz; j += blockDim.x) ysum[j] = pairwise_sum_masked(yb + (int64_t)j * ni, a.gas, ni);
  __syncthreads();
  // stencil-row spacing h_j: dz_ave inside, dzi at the two boundary rows
  auto h_of = [&](int j) {
    if (j == 0) return a.dzi[0];
    if (j == nz - 1) return a.dzi[nz - 2];
    return 0.5 * (a.dzi[j - 1] + a.dzi[j]);
  };
  if (g_Kzz) {
    for (int m = threadIdx.x; m < nz - 1; m += blockDim.x) {
      const double h0 = h_of(m), h1 = h_of(m + 1);
      const double ys0 = ysum[m], ys1 = ysum[m + 1];
      double dLdF = 0.0;
      for (int i = 0; i < ni; ++i) {
        const double grad = yb[(int64_t)(m + 1) * ni + i] / ys1 - yb[(int64_t)m * ni + i] / ys0;
        dLdF += grad * (lb[(int64_t)m * ni + i] / h0 - lb[(int64_t)(m + 1) * ni + i] / h1);
      }
      g_Kzz[g.z0 + m] = -dLdF * (ys1 + ys0) / (2.0 * a.dzi[m]);
    }
  }
  for (int i = threadIdx.x; i < ni; i += blockDim.x) {
    const int64_t o = (int64_t)b * ni + i;
    if (g_top) g_top[o] = (flags & VB_USE_TOPFLUX) ? -lb[(int64_t)(nz - 1) * ni + i] / a.dzi[nz - 2] : 0.0;
    if (g_bot) g_bot[o] = (flags & VB_USE_BOTFLUX) ? -lb[i] / a.dzi[0] : 0.0;
    if (g_vdep) g_vdep[o] = (flags & VB_USE_BOTFLUX) ? lb[i] * yb[i] / a.dzi[0] : 0.0;
  }
}

// ---- cotangents of every transport leaf of the atmosphere blob
// One stencil row's diffusion term (jax_step.py:67-246) of species i in flux
// form is (F of its upper interface - F of its lower one) / dz, with
//   F = (K+D)/d q + c D P + advection terms,   q = (y1s+y0s)/2 (y1/y1s - y0/y0s),
//   P = (-1/H + alpha/T (T1-T0)/d) (y0+y1) + ms/(Navo kb T) (g0 y0 + g1 y1)
// (0, 1: the layers below and above the interface; c = 1/2, 0 with vm; the end
// rows have one interface, its spacing as dz and their own gravity in both
// terms). Differentiated by hand in every leaf at once: one evaluation per
// (interface, species). An interface enters the two rows with opposite sign, so
// its leaves take the difference lambda_0/dz_0 - lambda_1/dz_1, formed first
// (RowPair): lambda is nearly conserved from layer to layer where the chemistry
// is slow, and the difference of the rows' products, each rounded, lost its
// digits (alpha against long double from the same lambda, median relative error:
// 2.8e-12 at 69 species and 17 layers with the rows apart, 1.2e-12 with dual
// numbers, 1.7e-13 so).
//
// CTA per block of VA_ROWS layers of an atmosphere, a warp per interface that
// enters their leaves (two more than the layers), lanes over species: the layer
// fields' derivatives are summed over species in the warp, the species' own are
// written at once, and every layer element then adds the one to three
// interfaces it enters, in a fixed order. FP64 arithmetic bound. ni=69, nz=120,
// 64 atmospheres (B200), both kernels: a thread per leaf element with dual
// numbers 12.8 ms (4 to 120 rows times up to 69 species each, 21.6 M
// evaluations), a warp per row 0.130 ms, now 0.089 (0.53 M evaluations).
constexpr int VA_ROWS = 8;
constexpr int VA_WARPS = VA_ROWS + 2;
// layer-field derivatives of an interface: Kzz, vz, Hpi, Ti, the spacing (not
// through dz), the temperature of the layer above (minus that of the one below),
// gravity of the layers below and above, lambda F / dz of the rows below and above
enum VaSlot { S_K, S_V, S_H, S_T, S_D, S_TCO, S_G0, S_G1, S_R0, S_R1, VA_SLOTS };

// The rows j and j + 1 that an interface enters: their dz, and
// lambda_j / dz_j - lambda_{j+1} / dz_{j+1} to a few roundings of its value.
struct RowPair {
  double rz0, rz1, rho, err;   // 1/dz of both, dz_j / dz_{j+1} and what it rounded off (over dz_{j+1})
  __device__ RowPair(const double* dzi, int nz, int j) {
    const double d = dzi[j], h0 = j == 0 ? d : 0.5 * (dzi[j - 1] + d), h1 = j == nz - 2 ? d : 0.5 * (d + dzi[j + 1]);
    rz0 = 1.0 / h0;
    rz1 = 1.0 / h1;
    rho = h0 / h1;
    err = fma(-rho, h1, h0) * rz1;
  }
  __device__ double diff(double l0, double l1) const { return (fma(-rho, l1, l0) - err * l1) * rz0; }
};

__host__ __device__ inline size_t vjp_atm_smem_bytes(int ni) {
  return ((size_t)(VA_ROWS + 3) * ni + ni + (VA_ROWS + 3) + VA_WARPS * VA_SLOTS) * sizeof(double);
}

__global__ void __launch_bounds__(VA_WARPS * 32)
vjp_atm_rows_kernel(Batch B, const double* __restrict__ y, const double* __restrict__ atm, int flags,
                    const double* __restrict__ lam, double* __restrict__ g_atm) {
  extern __shared__ double sm[];
  const int b = blockIdx.y, m0 = blockIdx.x * VA_ROWS;
  const Geo g = geo_of(B, b);
  const int ni = B.ni, nz = g.nz;
  if (m0 >= nz) return;
  const AtmRef a = atm_ref(atm + g.atm, nz, ni);
  const double* yb = y + g.z0 * ni;
  const double* lb = lam + g.z0 * ni;
  double* yr = sm;                                  // [VA_ROWS + 3][ni]: layers m0-1 ..
  double* gas = yr + (VA_ROWS + 3) * ni;
  double* ysum = gas + ni;                          // [VA_ROWS + 3]
  double* S = ysum + VA_ROWS + 3;                   // [VA_WARPS][VA_SLOTS]: interfaces m0-1 ..
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < (VA_ROWS + 3) * ni; e += VA_WARPS * 32) {
    const int jj = m0 - 1 + e / ni;
    yr[e] = (jj >= 0 && jj < nz) ? yb[(int64_t)(m0 - 1) * ni + e] : 0.0;
  }
  for (int i = threadIdx.x; i < ni; i += VA_WARPS * 32) gas[i] = a.gas[i];
  __syncthreads();
  // gas sums of the rows (0 outside the column, as the forward kernels)
  if (threadIdx.x < VA_ROWS + 3) {
    const int jj = m0 - 1 + (int)threadIdx.x;
    ysum[threadIdx.x] = (jj >= 0 && jj < nz) ? pairwise_sum_masked(yr + threadIdx.x * ni, gas, ni) : 0.0;
  }
  __syncthreads();
  const AtmOff o = atm_offsets(nz, ni);
  double* out = g_atm + g.atm;
  {
    const int q = m0 - 1 + warp;
    double acc[VA_SLOTS] = {};
    if (q >= 0 && q < nz - 1) {
      const bool lo = q == 0, hi = q == nz - 2, mine = q >= m0 && q < m0 + VA_ROWS;
      const double use_vm = (flags & VB_USE_VM_MOL) ? 1.0 : 0.0, use_set = (flags & VB_USE_SETTLING) ? 1.0 : 0.0;
      const double c = 0.5 * (1.0 - use_vm);
      const double *y0r = yr + warp * ni, *l0r = lb + (int64_t)q * ni;
      const double ys0 = ysum[warp], ys1 = ysum[warp + 1], half = 0.5 * (ys1 + ys0);
      const RowPair rows(a.dzi, nz, q);
      const double rd = 1.0 / a.dzi[q], K = a.Kzz[q], v = a.vz[q], rH = 1.0 / a.Hpi[q], rT = 1.0 / a.Ti[q];
      const double t = (a.Tco[q + 1] - a.Tco[q]) * rd, g0 = a.g[q], g1 = a.g[q + 1];
      // derivative of an advection term of interface speed v: upwind from below / above
      auto wind = [](double v, double below, double above) { return v > 0.0 ? below : (v < 0.0 ? above : 0.0); };
      for (int i = lane; i < ni; i += 32) {
        const int64_t at = (int64_t)q * ni + i;
        const double y0 = y0r[i], y1 = y0r[ni + i], l0 = l0r[i], l1 = l0r[ni + i];
        const double w0 = l0 * rows.rz0, w1 = l1 * rows.rz1, w = rows.diff(l0, l1);
        const double D = a.Dzz[at], al = a.alpha[i], mk = a.ms[i] / (NAVO * KB) * rT;
        const double vm0 = a.vm[at], vm1 = hi ? a.vm[at + ni] : vm0, vs = a.vs[at];   // the top row reads its own vm
        const double qd = half * (y1 / ys1 - y0 / ys0), s = y0 + y1;
        const double th = al * rT * t, Bt = th * s + mk * (g0 * y0 + g1 * y1), Pm = Bt - rH * s;
        const double e0 = lo ? mk * (g0 - g1) * y1 : 0.0, e1 = hi ? mk * (g1 - g0) * y0 : 0.0;   // end rows' gravity
        const double cD = c * D, cor = w0 * e0 - w1 * e1, wc = w * cD, gw = cD * mk;
        const double ez = -wind(v, y0, y1), em0 = -wind(vm0, y0, y1), em1 = -wind(vm1, y0, y1), es = -wind(vs, y0, y1);
        acc[S_K] += w * qd * rd;
        acc[S_V] += w * ez;
        acc[S_H] += wc * s * rH * rH;
        acc[S_T] -= (wc * Bt + cD * cor) * rT;
        acc[S_D] -= w * (K + D) * rd * rd * qd + wc * th * rd * s;
        acc[S_TCO] += wc * al * rT * rd * s;
        acc[S_G0] += gw * ((hi ? w0 : w) * y0 + (lo ? w0 * y1 : 0.0));
        acc[S_G1] += gw * ((lo ? -w1 : w) * y1 - (hi ? w1 * y0 : 0.0));
        const double F = (K + D) * rd * qd + v * ez + use_set * vs * es;
        acc[S_R0] += w0 * (F + cD * (Pm + e0) + use_vm * vm0 * em0);
        acc[S_R1] -= w1 * (F + cD * (Pm + e1) + use_vm * vm1 * em1);
        if (lo && (flags & VB_USE_BOTFLUX)) acc[S_D] -= l0 * (a.bot[i] - y0 * a.vdep[i]) * rd * rd;
        if (hi && (flags & VB_USE_TOPFLUX)) acc[S_D] -= l1 * a.top[i] * rd * rd;
        if (mine) {
          out[o.Dzz + at] = -(w * (qd * rd + c * Pm) + c * cor);
          out[o.vs + at] = -(use_set * w * es);
          out[o.vm + at] = -(use_vm * (hi ? w0 : w) * em0);
          if (hi) out[o.vm + at + ni] = use_vm * w1 * em1;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < VA_SLOTS; ++k) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], off);
    }
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < VA_SLOTS; ++k) S[warp * VA_SLOTS + k] = acc[k];
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 7 * VA_ROWS; e += VA_WARPS * 32) {
    const int f = e / VA_ROWS, l = e % VA_ROWS, m = m0 + l;
    const double *s0 = S + l * VA_SLOTS, *s1 = s0 + VA_SLOTS, *s2 = s1 + VA_SLOTS;   // interfaces m - 1, m, m + 1
    if (f < 4) {
      const int64_t off[4] = {o.Kzz, o.vz, o.Hpi, o.Ti};
      if (m < nz - 1) out[off[f] + m] = -s1[f];
    } else if (f == 4) {
      // the spacing itself, and as the dz (or half of it) of rows m and m + 1
      if (m < nz - 1) {
        const double c0 = m == 0 ? 1.0 / a.dzi[0] : 0.5 / (0.5 * (a.dzi[m - 1] + a.dzi[m]));
        const double c1 = m == nz - 2 ? 1.0 / a.dzi[m] : 0.5 / (0.5 * (a.dzi[m] + a.dzi[m + 1]));
        out[o.dzi + m] = -(s1[S_D] - c0 * (s0[S_R1] + s1[S_R0]) - c1 * (s1[S_R1] + s2[S_R0]));
      }
    } else if (m < nz) {
      if (f == 5)
        out[o.Tco + m] = -(s0[S_TCO] - s1[S_TCO]);
      else
        out[o.g + m] = -(s0[S_G1] + s1[S_G0]);
    }
  }
}

// The leaves with one element per species: ms and alpha (summed over the
// column's interfaces), the boundary fluxes and the deposition velocity. CTA
// per atmosphere, warps over interfaces, lanes over species.
__global__ void __launch_bounds__(VJP_THREADS)
vjp_atm_species_kernel(Batch B, const double* __restrict__ y, const double* __restrict__ atm, int flags,
                       const double* __restrict__ lam, double* __restrict__ g_atm) {
  constexpr int NWARP = VJP_THREADS / 32;
  __shared__ double red[2][NWARP][VB_MAX_NI];
  const int b = blockIdx.x;
  const Geo g = geo_of(B, b);
  const int ni = B.ni, nz = g.nz;
  const AtmRef a = atm_ref(atm + g.atm, nz, ni);
  const double* yb = y + g.z0 * ni;
  const double* lb = lam + g.z0 * ni;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double c = (flags & VB_USE_VM_MOL) ? 0.0 : 0.5;
  for (int i = lane; i < ni; i += 32) {
    double gms = 0.0, gal = 0.0;
    for (int q = warp; q < nz - 1; q += NWARP) {
      const int64_t at = (int64_t)q * ni + i;
      const RowPair rows(a.dzi, nz, q);
      const double y0 = yb[at], y1 = yb[at + ni], l0 = lb[at], l1 = lb[at + ni], w = rows.diff(l0, l1);
      const double D = c * a.Dzz[at] / a.Ti[q], g0 = a.g[q], g1 = a.g[q + 1];
      // the end rows' own gravity in both terms
      const double e0 = q == 0 ? l0 * rows.rz0 * (g0 - g1) * y1 : 0.0;
      const double e1 = q == nz - 2 ? l1 * rows.rz1 * (g1 - g0) * y0 : 0.0;
      gms += D * (w * (g0 * y0 + g1 * y1) + (e0 - e1));
      gal += D * ((a.Tco[q + 1] - a.Tco[q]) / a.dzi[q]) * (y0 + y1) * w;
    }
    red[0][warp][i] = gms;
    red[1][warp][i] = gal;
  }
  __syncthreads();
  const AtmOff o = atm_offsets(nz, ni);
  double* out = g_atm + g.atm;
  for (int i = threadIdx.x; i < ni; i += VJP_THREADS) {
    double gms = 0.0, gal = 0.0;
#pragma unroll
    for (int q = 0; q < NWARP; ++q) {
      gms += red[0][q][i];
      gal += red[1][q][i];
    }
    out[o.ms + i] = -gms / (NAVO * KB);
    out[o.alpha + i] = -gal;
    // (no boundary flux: 0 lambda, so that a lambda that is not finite shows here too)
    const double lt = lb[(int64_t)(nz - 1) * ni + i], l0 = lb[i];
    out[o.top + i] = (flags & VB_USE_TOPFLUX) ? -lt / a.dzi[nz - 2] : -(0.0 * lt);
    out[o.bot + i] = (flags & VB_USE_BOTFLUX) ? -l0 / a.dzi[0] : -(0.0 * l0);
    out[o.vdep + i] = (flags & VB_USE_BOTFLUX) ? l0 * yb[i] / a.dzi[0] : -(0.0 * l0);
  }
}

// Copy the workspace's first-stage rows (k1: the adjoint's lambda, or the
// Ros2 step's k1) and, with k2 != nullptr, the Ros2 step's second-stage rows
// (kept in the aux rows by the final back sweep) into [layers][ni] arrays.
__global__ void gather_stages_kernel(Batch B, const double* __restrict__ ws, double* __restrict__ k1,
                                     double* __restrict__ k2) {
  const int b = blockIdx.y, j = blockIdx.x;
  Geo g = geo_of(B, b);
  if (j >= g.nz) return;
  WsView w = ws_view(const_cast<double*>(ws), g, B.ni, B.ld);
  const int64_t src = (int64_t)j * B.ni, dst = g.z0 * B.ni + (int64_t)j * B.ni;
  for (int i = threadIdx.x; i < B.ni; i += blockDim.x) {
    if (k1) k1[dst + i] = w.k1[src + i];
    if (k2) k2[dst + i] = w.aux[src + i];
  }
}

cudaError_t launch_gather_stages(const Batch& B, const double* ws, double* k1, double* k2, cudaStream_t st) {
  if (!k1 && !k2) return cudaSuccess;
  dim3 grid(B.nz, B.count);
  gather_stages_kernel<<<grid, 128, 0, st>>>(B, ws, k1, k2);
  return cudaGetLastError();
}

cudaError_t launch_vjp_atm(const Batch& B, const double* y, const double* atm, int flags, const double* lam,
                           double* g_atm, cudaStream_t st) {
  const size_t sm = vjp_atm_smem_bytes(B.ni);
  cudaError_t e = cudaFuncSetAttribute(vjp_atm_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  dim3 grid((B.nz + VA_ROWS - 1) / VA_ROWS, B.count);
  vjp_atm_rows_kernel<<<grid, VA_WARPS * 32, sm, st>>>(B, y, atm, flags, lam, g_atm);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  vjp_atm_species_kernel<<<B.count, VJP_THREADS, 0, st>>>(B, y, atm, flags, lam, g_atm);
  return cudaGetLastError();
}

cudaError_t launch_vjp(const NetDev& net, const Batch& B, const double* y, const double* k, const double* atm,
                       int flags, double* ws, double* g_k, double* g_M, double* g_Kzz, double* g_top,
                       double* g_bot, double* g_vdep, cudaStream_t st) {
  if (g_k || g_M) {
    dim3 grid(B.nz, B.count);
    vjp_k_kernel<<<grid, VJP_THREADS, 0, st>>>(net, B, y, k, atm, ws, g_k, g_M);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (g_Kzz || g_top || g_bot || g_vdep) {
    size_t sm = (size_t)B.nz * sizeof(double);
    vjp_transport_kernel<<<B.count, VJP_THREADS, sm, st>>>(B, y, atm, flags, ws, g_Kzz, g_top, g_bot, g_vdep);
    return cudaGetLastError();
  }
  return cudaSuccess;
}

}  // namespace vb
