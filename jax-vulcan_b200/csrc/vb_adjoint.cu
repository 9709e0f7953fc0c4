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
// form, F = E / dz with
//   E = (K2+D2)/d2 q2 - (K1+D1)/d1 q1 + c (D2 P2 - D1 P1) + advection terms,
//   q2 = (ysp+ys0)/2 (yp/ysp - y0/ys0),   q1 = (ys0+ysm)/2 (y0/ys0 - ym/ysm),
//   P2 = (-1/H2 + alpha/T2 (Tp-T0)/d2) (y0+yp) + ms/(Navo kb T2) (g0 y0 + gp yp)
// (2: the interface above, j; 1: the one below, j-1; c = 1/2, 0 with vm; the
// end rows have one interface, its spacing as dz and their own gravity in both
// terms), differentiated by hand in every leaf at once: one evaluation per
// (row, species) instead of one per leaf element, row and species.
//
// CTA per block of VA_ROWS layers of an atmosphere, a warp per stencil row that
// enters them (two more than the layers), lanes over species: the layer fields'
// derivatives are summed over species in the warp, the species' own go to
// shared memory, and every leaf element then adds the two or three rows it
// enters, in a fixed order. FP64 arithmetic bound (about 20 divisions a row and
// species). ni=69, nz=120, 64 atmospheres (B200): a thread per leaf element
// with dual numbers 12.8 ms (4 to 120 rows times up to 69 species each, 21.6 M
// evaluations), the two kernels below 0.077 and 0.064 ms (0.66 M evaluations of the rows).
constexpr int VA_ROWS = 8;
constexpr int VA_WARPS = VA_ROWS + 2;
constexpr int VA_SLOTS = 16;   // layer-field derivatives of a row (VaSlot)
enum VaSlot { S_K2, S_K1, S_D2, S_D1, S_V2, S_V1, S_H2, S_H1, S_T2, S_T1, S_TM, S_T0, S_TP, S_GM, S_G0, S_GP };
constexpr int VA_SPEC = 6;     // species' own: Dzz, vm, vs at j and at j-1

__host__ __device__ inline size_t vjp_atm_smem_bytes(int ni) {
  return ((size_t)(VA_ROWS + 4) * ni + ni + (VA_ROWS + 4) + VA_WARPS * VA_SLOTS + (size_t)VA_WARPS * VA_SPEC * ni) *
         sizeof(double);
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
  double* yr = sm;                                  // [VA_ROWS + 4][ni]: layers m0-2 ..
  double* gas = yr + (VA_ROWS + 4) * ni;
  double* ysum = gas + ni;                          // [VA_ROWS + 4]
  double* S = ysum + VA_ROWS + 4;                   // [VA_WARPS][VA_SLOTS]: rows m0-1 ..
  double* P = S + VA_WARPS * VA_SLOTS;              // [VA_WARPS][VA_SPEC][ni]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < (VA_ROWS + 4) * ni; e += VA_WARPS * 32) {
    const int jj = m0 - 2 + e / ni;
    yr[e] = (jj >= 0 && jj < nz) ? yb[(int64_t)(m0 - 2) * ni + e] : 0.0;
  }
  for (int i = threadIdx.x; i < ni; i += VA_WARPS * 32) gas[i] = a.gas[i];
  __syncthreads();
  // gas sums of the rows (0 outside the column, as the forward kernels)
  if (threadIdx.x < VA_ROWS + 4) {
    const int jj = m0 - 2 + (int)threadIdx.x;
    ysum[threadIdx.x] = (jj >= 0 && jj < nz) ? pairwise_sum_masked(yr + threadIdx.x * ni, gas, ni) : 0.0;
  }
  __syncthreads();
  {
    const int j = m0 - 1 + warp;
    const bool row = j >= 0 && j < nz, up = row && j < nz - 1, dn = row && j > 0;
    double acc[VA_SLOTS] = {};
    if (row) {
      const double use_vm = (flags & VB_USE_VM_MOL) ? 1.0 : 0.0, use_set = (flags & VB_USE_SETTLING) ? 1.0 : 0.0;
      const double c = 0.5 * (1.0 - use_vm);
      const double* y0r = yr + (warp + 1) * ni;
      const double ys0 = ysum[warp + 1], ysm = ysum[warp], ysp = ysum[warp + 2];
      const double d2 = up ? a.dzi[j] : 0.0, d1 = dn ? a.dzi[j - 1] : 0.0;
      const double rz = (up && dn) ? 1.0 / (0.5 * (d1 + d2)) : 1.0 / (up ? d2 : d1);
      const double drz = (up && dn) ? -0.5 * rz : -rz;   // d(1/dz)/d(spacing) = drz / dz
      const double K2 = up ? a.Kzz[j] : 0.0, K1 = dn ? a.Kzz[j - 1] : 0.0;
      const double v2 = up ? a.vz[j] : 0.0, v1 = dn ? a.vz[j - 1] : 0.0;
      const double rH2 = up ? 1.0 / a.Hpi[j] : 0.0, rH1 = dn ? 1.0 / a.Hpi[j - 1] : 0.0;
      const double rT2 = up ? 1.0 / a.Ti[j] : 0.0, rT1 = dn ? 1.0 / a.Ti[j - 1] : 0.0;
      const double rd2 = up ? 1.0 / d2 : 0.0, rd1 = dn ? 1.0 / d1 : 0.0;
      const double T0 = a.Tco[j];
      const double t2 = up ? (a.Tco[j + 1] - T0) * rd2 : 0.0, t1 = dn ? (T0 - a.Tco[j - 1]) * rd1 : 0.0;
      const double g0 = a.g[j], gp = (up && dn) ? a.g[j + 1] : g0, gm = (up && dn) ? a.g[j - 1] : g0;
      const double S2 = 0.5 * (ysp + ys0), S1 = 0.5 * (ys0 + ysm);
      for (int i = lane; i < ni; i += 32) {
        const double y0 = y0r[i], yp = y0r[ni + i], ym = y0r[i - ni];
        const double L = lb[(int64_t)j * ni + i], w = L * rz;
        const double al = a.alpha[i], mk = a.ms[i] / (NAVO * KB);
        double E = 0.0, sp[VA_SPEC] = {};
        // derivative of an advection term of interface speed v: upwind from below / above
        auto wind = [](double v, double below, double above) { return v > 0.0 ? below : (v < 0.0 ? above : 0.0); };
        if (up) {
          const double D2 = a.Dzz[(int64_t)j * ni + i], vm = a.vm[(int64_t)j * ni + i], vs = a.vs[(int64_t)j * ni + i];
          const double q = S2 * (yp / ysp - y0 / ys0), s = y0 + yp, gy = g0 * y0 + gp * yp;
          const double th = al * rT2 * t2, Pm = (th - rH2) * s + mk * rT2 * gy;
          const double wc = w * c * D2, th_w = wc * al * rT2 * rd2 * s, gw = wc * mk * rT2;
          E += (K2 + D2) * rd2 * q + c * D2 * Pm;
          acc[S_K2] += w * q * rd2;
          sp[0] = w * (q * rd2 + c * Pm);
          acc[S_H2] += wc * s * rH2 * rH2;
          acc[S_T2] -= wc * (th * s + mk * rT2 * gy) * rT2;
          acc[S_TP] += th_w;
          acc[S_T0] -= th_w;
          acc[S_G0] += gw * y0;
          acc[dn ? S_GP : S_G0] += gw * yp;
          acc[S_D2] -= w * (K2 + D2) * rd2 * rd2 * q + wc * th * rd2 * s;
          const double ez = -wind(v2, y0, yp), em = -wind(vm, y0, yp), es = -wind(vs, y0, yp);
          acc[S_V2] += w * ez;
          sp[2] = use_vm * w * em;
          sp[4] = use_set * w * es;
          E += v2 * ez + use_vm * vm * em + use_set * vs * es;
        }
        if (dn) {
          const int64_t mv = (int64_t)(up ? j - 1 : j) * ni + i;   // the top row reads its own vm
          const double D1 = a.Dzz[(int64_t)(j - 1) * ni + i], vm = a.vm[mv], vs = a.vs[(int64_t)(j - 1) * ni + i];
          const double q = S1 * (y0 / ys0 - ym / ysm), s = y0 + ym, gy = g0 * y0 + gm * ym;
          const double th = al * rT1 * t1, Pm = (th - rH1) * s + mk * rT1 * gy;
          const double wc = w * c * D1, th_w = wc * al * rT1 * rd1 * s, gw = wc * mk * rT1;
          E -= (K1 + D1) * rd1 * q + c * D1 * Pm;
          acc[S_K1] -= w * q * rd1;
          sp[1] = -w * (q * rd1 + c * Pm);
          acc[S_H1] -= wc * s * rH1 * rH1;
          acc[S_T1] += wc * (th * s + mk * rT1 * gy) * rT1;
          acc[S_TM] += th_w;
          acc[S_T0] -= th_w;
          acc[S_G0] -= gw * y0;
          acc[up ? S_GM : S_G0] -= gw * ym;
          acc[S_D1] += w * (K1 + D1) * rd1 * rd1 * q + wc * th * rd1 * s;
          const double ez = wind(v1, ym, y0), em = wind(vm, ym, y0), es = wind(vs, ym, y0);
          acc[S_V1] += w * ez;
          sp[up ? 3 : 2] += use_vm * w * em;
          sp[5] = use_set * w * es;
          E += v1 * ez + use_vm * vm * em + use_set * vs * es;
        }
        const double dF = L * drz * rz * E;
        if (up) acc[S_D2] += dF;
        if (dn) acc[S_D1] += dF;
        if (j == 0 && (flags & VB_USE_BOTFLUX)) acc[S_D2] -= L * (a.bot[i] - y0 * a.vdep[i]) * rd2 * rd2;
        if (j == nz - 1 && (flags & VB_USE_TOPFLUX)) acc[S_D1] -= L * a.top[i] * rd1 * rd1;
#pragma unroll
        for (int q = 0; q < VA_SPEC; ++q) P[(warp * VA_SPEC + q) * ni + i] = sp[q];
      }
    } else {
      for (int e = lane; e < VA_SPEC * ni; e += 32) P[warp * VA_SPEC * ni + e] = 0.0;
    }
#pragma unroll
    for (int q = 0; q < VA_SLOTS; ++q) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], off);
    }
    if (lane == 0) {
#pragma unroll
      for (int q = 0; q < VA_SLOTS; ++q) S[warp * VA_SLOTS + q] = acc[q];
    }
  }
  __syncthreads();
  const AtmOff o = atm_offsets(nz, ni);
  double* out = g_atm + g.atm;
  for (int e = threadIdx.x; e < 7 * VA_ROWS; e += VA_WARPS * 32) {
    const int f = e / VA_ROWS, l = e % VA_ROWS, m = m0 + l;
    const double* s = S + l * VA_SLOTS;   // row m - 1; rows m and m + 1 follow
    if (f < 5) {
      const int64_t off[5] = {o.Kzz, o.dzi, o.vz, o.Hpi, o.Ti};
      if (m < nz - 1) out[off[f] + m] = -(s[VA_SLOTS + 2 * f] + s[2 * VA_SLOTS + 2 * f + 1]);
    } else if (m < nz) {
      const int q = f == 5 ? S_TM : S_GM;   // j-1, j, j+1 of the field
      out[(f == 5 ? o.Tco : o.g) + m] = -(s[q + 2] + s[VA_SLOTS + q + 1] + s[2 * VA_SLOTS + q]);
    }
  }
  for (int e = threadIdx.x; e < VA_ROWS * ni; e += VA_WARPS * 32) {
    const int l = e / ni, i = e - l * ni, m = m0 + l;
    if (m >= nz) break;
    const double* r0 = P + (l + 1) * VA_SPEC * ni + i;   // row m
    const double* r1 = r0 + VA_SPEC * ni;                // row m + 1
    const int64_t at = (int64_t)m * ni + i;
    if (m < nz - 1) {
      out[o.Dzz + at] = -(r0[0] + r1[ni]);
      out[o.vs + at] = -(r0[4 * ni] + r1[5 * ni]);
    }
    out[o.vm + at] = -(r0[2 * ni] + r1[3 * ni]);
  }
}

// The leaves with one element per species: ms and alpha (summed over the
// column), the boundary fluxes and the deposition velocity. CTA per atmosphere,
// warps over rows, lanes over species.
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
    for (int j = warp; j < nz; j += NWARP) {
      const bool up = j < nz - 1, dn = j > 0;
      const double d2 = up ? a.dzi[j] : 0.0, d1 = dn ? a.dzi[j - 1] : 0.0;
      const double dz = (up && dn) ? 0.5 * (d1 + d2) : (up ? d2 : d1);
      const double w = c * lb[(int64_t)j * ni + i] / dz, y0 = yb[(int64_t)j * ni + i], g0 = a.g[j];
      if (up) {
        const double yp = yb[(int64_t)(j + 1) * ni + i], D = w * a.Dzz[(int64_t)j * ni + i] / a.Ti[j];
        gms += D * (g0 * y0 + (dn ? a.g[j + 1] : g0) * yp);
        gal += D * ((a.Tco[j + 1] - a.Tco[j]) / d2) * (y0 + yp);
      }
      if (dn) {
        const double ym = yb[(int64_t)(j - 1) * ni + i], D = w * a.Dzz[(int64_t)(j - 1) * ni + i] / a.Ti[j - 1];
        gms -= D * (g0 * y0 + (up ? a.g[j - 1] : g0) * ym);
        gal -= D * ((a.Tco[j] - a.Tco[j - 1]) / d1) * (y0 + ym);
      }
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
    out[o.top + i] = (flags & VB_USE_TOPFLUX) ? -lb[(int64_t)(nz - 1) * ni + i] / a.dzi[nz - 2] : 0.0;
    out[o.bot + i] = (flags & VB_USE_BOTFLUX) ? -lb[i] / a.dzi[0] : 0.0;
    out[o.vdep + i] = (flags & VB_USE_BOTFLUX) ? lb[i] * yb[i] / a.dzi[0] : 0.0;
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
