// Photochemistry kernels (reference photo.py):
//   tau_kernel   optical depth, a top-down running sum per wavelength bin
//                (photo.py:84-123);
//   flux_kernel  two-stream Eddington flux: coefficients of every layer in
//                parallel, the down and the up recursions in z in one thread
//                per bin (photo.py:126-245);
//   j_kernel     J-rates of a tile of layers and every branch, warp per
//                branch, reductions over bins with the two-resolution
//                trapezoid correction, fused with the write of the photolysis
//                rows of k (photo.py:309-351, 455-478).
// Each kernel takes an optional per-atmosphere mask `due` (atmospheres with
// due[b] == 0 are left alone: the photo branch of the adaptive loop runs only
// where its cadence says so, outer_loop.py:716-724), and the flux kernel an
// optional per-atmosphere accumulator of the actinic-flux change
// (outer_loop.py:327-336), which the tau kernel of the same update zeroes.
// Compiled with --fmad=false: products and sums round as the reference's
// element-wise expressions do.
#include <cuda_runtime.h>

#include <algorithm>

#include "vb_common.cuh"
#include "vb_launch.cuh"

namespace vb {

constexpr int PHOTO_THREADS = 128;
// achg points at VbConvState::aflux_change of atmosphere 0; the records are
// VbConvState-sized apart
constexpr int64_t ACHG_STRIDE = sizeof(VbConvState) / sizeof(double);
static_assert(sizeof(VbConvState) % sizeof(double) == 0, "VbConvState size");

// Tiled kernels (tau_kernel, flux_kernel): a CTA takes PB bins of one
// atmosphere and all its layers. Everything that does not depend on the layer
// before (absorber sums, exponentials, roots, divisions) runs with a thread per
// (layer, bin) into shared memory; only the recursions in z run with one thread
// per bin, from operands loaded ahead, and all threads write the results. The
// arithmetic of each value is the reference's, in its order. One thread per bin
// for the whole column left a chain of 120 layers x ~300 dependent FP64
// instructions per thread, and 20 CTAs on 148 SMs for one atmosphere.
// 32 bins a tile: the recursion, which one warp runs while the others wait,
// serves 32 bins at a time; the flux tile's seven rows per layer then fill one
// SM's shared memory at nz = 120. nz=120, 2500 bins, 40 branches (B200, us,
// before -> now, launches back to back): tau 1 atmosphere 261 -> 11, 64: 403 ->
// 208; flux 449 -> 27, 1412 -> 967 (about 220 FP64 instructions per layer and
// bin; the recursion's share is a quarter); J (below) 33 -> 21, 570 -> 267.
constexpr size_t PHOTO_SMEM_MAX = 220 * 1024;

// Cross sections of the tile's bins (absorbers, then scatterers; 0 outside nbin)
// in shared memory, [n_abs + n_scat][PB].
template <int PB>
__host__ __device__ inline size_t tile_table_doubles(const VbPhoto& P) {
  return (size_t)(P.n_abs + P.n_scat) * PB;
}
template <int PB, int PT>
__device__ inline void load_cross(const VbPhoto& P, double* cs, int bin0) {
  for (int e = threadIdx.x; e < (P.n_abs + P.n_scat) * PB; e += PT) {
    const int k = e / PB, bin = bin0 + e % PB;
    double v = 0.0;
    if (bin < P.nbin)
      v = k < P.n_abs ? P.absp_cross[(int64_t)k * P.nbin + bin] : P.scat_cross[(int64_t)(k - P.n_abs) * P.nbin + bin];
    cs[e] = v;
  }
}
// Weights of a column's layers by species in table order (absorbers,
// temperature-dependent absorbers, scatterers), [nz][n].
template <int PT>
__device__ inline void load_weights(const VbPhoto& P, double* wt, const double* __restrict__ w, int nz, int ni) {
  const int n = P.n_abs + P.n_abs_T + P.n_scat;
  for (int k = threadIdx.x & 31; k < n; k += 32) {   // lanes over species, warps over layers
    const int i = k < P.n_abs ? P.absp_idx[k] : k < P.n_abs + P.n_abs_T ? P.absp_T_idx[k - P.n_abs]
                                                                        : P.scat_idx[k - P.n_abs - P.n_abs_T];
#pragma unroll 8
    for (int j = threadIdx.x >> 5; j < nz; j += PT / 32) wt[j * n + k] = w[(int64_t)j * ni + i];
  }
}

// Species-weighted cross-section sums of JL layers j, j + PR, .. (those below
// nz) of one bin (c = bin in the tile): absorbers, temperature-dependent
// absorbers, scatterers, each in table order. Four layers share a cross
// section's load: with one layer at a time the loads (three per term) bounded
// the tile.
constexpr int JL = 4;
template <int PB, int PR>
__device__ __forceinline__ void column_sums(const VbPhoto& P, const double* cs, const double* wt,
                                            const double* __restrict__ xT, int nz, int j, int bin, int c,
                                            double (&sa)[JL], double (&sT)[JL], double (&ss)[JL]) {
  const int n = P.n_abs + P.n_abs_T + P.n_scat;
  const double* w[JL];
  const double* x[JL];
#pragma unroll
  for (int l = 0; l < JL; ++l) {
    const int jl = min(j + l * PR, nz - 1);   // beyond the column: a repeat nobody reads
    w[l] = wt + jl * n;
    x[l] = xT + (int64_t)jl * P.nbin + bin;
    sa[l] = sT[l] = ss[l] = 0.0;
  }
  cs += c;
#pragma unroll 2
  for (int k = 0; k < P.n_abs; ++k) {
    const double v = cs[k * PB];
#pragma unroll
    for (int l = 0; l < JL; ++l) sa[l] = sa[l] + w[l][k] * v;
  }
  const int64_t tstep = (int64_t)nz * P.nbin;
#pragma unroll 2
  for (int k = 0; k < P.n_abs_T; ++k)
#pragma unroll
    for (int l = 0; l < JL; ++l) sT[l] = sT[l] + w[l][P.n_abs + k] * x[l][k * tstep];
  cs += P.n_abs * PB;
  for (int k = 0; k < P.n_scat; ++k) {
    const double v = cs[k * PB];
#pragma unroll
    for (int l = 0; l < JL; ++l) ss[l] = ss[l] + w[l][P.n_abs + P.n_abs_T + k] * v;
  }
}

template <int PB>
__host__ __device__ inline size_t tau_smem_bytes(const VbPhoto& P, int nz) {
  return ((size_t)nz * (PB + P.n_abs + P.n_abs_T + P.n_scat) + tile_table_doubles<PB>(P)) * sizeof(double);
}

template <int PB, int PT>
__global__ void __launch_bounds__(PT, 1024 / PT)
tau_kernel(int nz, int ni, VbPhoto P, const double* __restrict__ y, const double* __restrict__ dz,
           double* __restrict__ tau, const int32_t* __restrict__ due, double* __restrict__ achg) {
  constexpr int PR = PT / PB;   // layers in flight
  extern __shared__ double smp[];
  const int b = blockIdx.y, bin0 = blockIdx.x * PB;
  if (due && due[b] == 0) return;
  if (achg && blockIdx.x == 0 && threadIdx.x == 0) achg[(int64_t)b * ACHG_STRIDE] = 0.0;
  const int nbin = P.nbin, c = threadIdx.x % PB, bin = bin0 + c;
  const bool on = bin < nbin;
  double* a = smp;   // [nz][PB]: the layers' depths, then their running sum
  double* cs = a + nz * PB;
  double* wt = cs + tile_table_doubles<PB>(P);
  load_cross<PB, PT>(P, cs, bin0);
  load_weights<PT>(P, wt, y + (int64_t)b * nz * ni, nz, ni);
  __syncthreads();
  const double* dzb = dz + (int64_t)b * nz;
  const double* xT = P.absp_T_cross + (int64_t)b * P.T_stride;
  double* tb = tau + (int64_t)b * (nz + 1) * nbin;
  for (int j0 = threadIdx.x / PB; j0 < nz && on; j0 += JL * PR) {
    double sa[JL], sT[JL], ss[JL];
    column_sums<PB, PR>(P, cs, wt, xT, nz, j0, bin, c, sa, sT, ss);
#pragma unroll
    for (int l = 0; l < JL; ++l) {
      const int j = j0 + l * PR;
      if (j < nz) {
        double v = 0.0;
        if (P.n_abs > 0) v = sa[l] * dzb[j];
        if (P.n_abs_T > 0) v = v + sT[l] * dzb[j];
        if (P.n_scat > 0) v = v + ss[l] * dzb[j];
        a[j * PB + c] = v;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < PB && on) {
    // eight layers' depths at a time in registers: the chain is one addition a layer
    double acc = a[(nz - 1) * PB + c];
    int j = nz - 2;
    for (; j >= 7; j -= 8) {
      double v[8];
#pragma unroll
      for (int l = 0; l < 8; ++l) v[l] = a[(j - l) * PB + c];
#pragma unroll
      for (int l = 0; l < 8; ++l) {
        acc = acc + v[l];
        a[(j - l) * PB + c] = acc;
      }
    }
    for (; j >= 0; --j) {
      acc = acc + a[j * PB + c];
      a[j * PB + c] = acc;
    }
  }
  __syncthreads();
  if (on)
    for (int j = threadIdx.x / PB; j <= nz; j += PR) tb[(int64_t)j * nbin + bin] = j < nz ? a[j * PB + c] : 0.0;
}

// The same with a thread per bin and column: columns whose tile does not fit
// shared memory, and many short ones (short_columns).
__global__ void __launch_bounds__(PHOTO_THREADS)
tau_column_kernel(int nz, int ni, VbPhoto P, const double* __restrict__ y, const double* __restrict__ dz,
           double* __restrict__ tau, const int32_t* __restrict__ due, double* __restrict__ achg) {
  const int b = blockIdx.y;
  const int bin = blockIdx.x * blockDim.x + threadIdx.x;
  if (due && due[b] == 0) return;
  if (achg && bin == 0) achg[(int64_t)b * ACHG_STRIDE] = 0.0;
  if (bin >= P.nbin) return;
  const int nbin = P.nbin;
  const double* yb = y + (int64_t)b * nz * ni;
  const double* dzb = dz + (int64_t)b * nz;
  const double* xT = P.absp_T_cross + (int64_t)b * P.T_stride;
  double* tb = tau + (int64_t)b * (nz + 1) * nbin;
  tb[(int64_t)nz * nbin + bin] = 0.0;
  double acc = 0.0;
  for (int j = nz - 1; j >= 0; --j) {
    const double* yj = yb + (int64_t)j * ni;
    double a = 0.0;
    if (P.n_abs > 0) {
      double s = 0.0;
      for (int k = 0; k < P.n_abs; ++k) s = s + yj[P.absp_idx[k]] * P.absp_cross[(int64_t)k * nbin + bin];
      a = s * dzb[j];
    }
    if (P.n_abs_T > 0) {
      double s = 0.0;
      for (int k = 0; k < P.n_abs_T; ++k)
        s = s + yj[P.absp_T_idx[k]] * xT[((int64_t)k * nz + j) * nbin + bin];
      a = a + s * dzb[j];
    }
    if (P.n_scat > 0) {
      double s = 0.0;
      for (int k = 0; k < P.n_scat; ++k) s = s + yj[P.scat_idx[k]] * P.scat_cross[(int64_t)k * nbin + bin];
      a = a + s * dzb[j];
    }
    acc = (j == nz - 1) ? a : acc + a;
    tb[(int64_t)j * nbin + bin] = acc;
  }
}

struct TwoStream {
  double chi, xi, phi, gp, gm;
};

// w0 = scat / (abs + scat), NaN -> 0, at most 1 - 1e-8 (photo.py:166-170).
__device__ __forceinline__ double albedo_of(double tot_abs, double tot_scat) {
  double w0 = tot_scat / fmax(tot_abs + tot_scat, 1e-300);
  if (isnan(w0)) w0 = 0.0;
  return fmin(w0, 1.0 - 1e-8);
}

// Single-scattering albedo of one layer and bin (photo.py:150-170): the
// ymix-weighted absorption (T-independent and T-dependent cross sections)
// and scattering sums, w0 = scat / (abs + scat), NaN -> 0, at most 1 - 1e-8.
__device__ inline double albedo(const VbPhoto& P, const double* __restrict__ xT, int nz, const double* ymix_j, int j,
                                int bin) {
  const int nbin = P.nbin;
  double tot_abs = 0.0, tot_scat = 0.0;
  if (P.n_abs > 0) {
    double s = 0.0;
    for (int k = 0; k < P.n_abs; ++k) s = s + ymix_j[P.absp_idx[k]] * P.absp_cross[(int64_t)k * nbin + bin];
    tot_abs = s;
  }
  if (P.n_abs_T > 0) {
    double s = 0.0;
    for (int k = 0; k < P.n_abs_T; ++k)
      s = s + ymix_j[P.absp_T_idx[k]] * xT[((int64_t)k * nz + j) * nbin + bin];
    tot_abs = tot_abs + s;
  }
  if (P.n_scat > 0) {
    double s = 0.0;
    for (int k = 0; k < P.n_scat; ++k) s = s + ymix_j[P.scat_idx[k]] * P.scat_cross[(int64_t)k * nbin + bin];
    tot_scat = s;
  }
  return albedo_of(tot_abs, tot_scat);
}

// The quotients of the two-stream formulas that depend on the atmosphere's
// angles only, formed once per thread.
struct StreamConst {
  double mu, neg_redd, rmu2, redd2, redd, sum, dif;
  __device__ explicit StreamConst(const VbPhoto& P)
      : mu(-1.0 * P.mu_zenith), neg_redd(-1.0 / P.edd), rmu2(1.0 / (mu * mu)), redd2(1.0 / (P.edd * P.edd)),
        redd(1.0 / P.edd), sum(redd + 1.0 / mu), dif(redd - 1.0 / mu) {}
};

// Two-stream coefficients of one layer from its albedo (photo.py:171-203).
__device__ inline TwoStream two_stream(const VbPhoto& P, const StreamConst& k, double w0, double dtau) {
  const double ag0 = P.ag0;
  double tran, zp, zm, ll, gp, gm;
  if (ag0 == 0.0) {
    const double sq = sqrt(1.0 - w0);
    tran = exp(k.neg_redd * sq * dtau);
    zp = 0.5 * (1.0 + sq);
    zm = 0.5 * (1.0 - sq);
    ll = -1.0 * w0 / (k.rmu2 - k.redd2 * (1.0 - w0));
    gp = 0.5 * (ll * k.sum);
    gm = 0.5 * (ll * k.dif);
  } else {
    const double wa = 1.0 - w0 * ag0;
    tran = exp(k.neg_redd * sqrt(wa * (1.0 - w0)) * dtau);
    const double rt = sqrt((1.0 - w0) / wa);
    zp = 0.5 * (1.0 + rt);
    zm = 0.5 * (1.0 - rt);
    ll = ((1.0 - w0) * wa - 1.0) / (k.rmu2 - k.redd2 * (1.0 - w0) * wa);
    gp = 0.5 * (ll * (k.redd + 1.0 / (k.mu * wa)) + w0 * ag0 * k.mu / wa);
    gm = 0.5 * (ll * (k.redd - 1.0 / (k.mu * wa)) - w0 * ag0 * k.mu / wa);
  }
  TwoStream c;
  c.chi = zm * zm * (tran * tran) - zp * zp;
  c.xi = zp * zm * (1.0 - tran * tran);
  c.phi = (zm * zm - zp * zp) * tran;
  c.gp = gp;
  c.gm = gm;
  return c;
}

// Rows per layer of the flux tile: phi, xi, 1/chi, the upward flux of the
// previous call (then the downward flux), i_d/mu (then the upward flux), i_u/mu
// and the direct beam of the nz + 1 levels.
template <int PB>
__host__ __device__ inline size_t flux_smem_bytes(const VbPhoto& P, int nz) {
  return ((size_t)(7 * nz + 1) * PB + tile_table_doubles<PB>(P)) * sizeof(double);
}
// the weights' tile lies over the rows xi and 1/chi until the coefficients are formed
template <int PB>
constexpr int FLUX_MAX_SPECIES = 2 * PB;
constexpr int FLUX_THREADS = 512;   // of an SM: 128 registers each

template <int PB, int PT>
__global__ void __launch_bounds__(PT, FLUX_THREADS / PT)
flux_kernel(int nz, int ni, VbPhoto P, const double* __restrict__ tau, const double* __restrict__ ymix,
            const double* du_prev, double* __restrict__ aflux, double* __restrict__ sflux,
            double* __restrict__ dd, double* du, const int32_t* __restrict__ due, double flux_atol,
            double* __restrict__ achg) {
  // du_prev and du may be one buffer: the tile's bins of du_prev are read
  // before the block writes du.
  constexpr int PR = PT / PB;   // layers in flight
  extern __shared__ double smp[];
  const int b = blockIdx.y, bin0 = blockIdx.x * PB;
  if (due && due[b] == 0) return;
  const int nbin = P.nbin, c = threadIdx.x % PB, bin = bin0 + c, row = threadIdx.x / PB;
  const bool on = bin < nbin;
  const int L = nz * PB;
  double* phi = smp + c;
  double *xi = phi + L, *rc = xi + L, *ud = rc + L, *id = ud + L, *iu = id + L, *sb = iu + L;
  double* cs = smp + (7 * nz + 1) * PB;
  double* wt = smp + L;
  const int64_t zb = (int64_t)b * (nz + 1) * nbin + bin;
  const double* tb = tau + zb;
  // the optical depths (parked in the i_u row) and dflux_u of the previous call
  // come in while the tables are loaded
  if (on)
    for (int j = row; j < nz; j += PR) {
      cp_async8(iu + j * PB, tb + (int64_t)j * nbin);
      cp_async8(ud + j * PB, du_prev + zb + (int64_t)j * nbin);
    }
  load_cross<PB, PT>(P, cs, bin0);
  load_weights<PT>(P, wt, ymix + (int64_t)b * nz * ni, nz, ni);
  const double* xT = P.absp_T_cross + (int64_t)b * P.T_stride;
  const StreamConst sc(P);
  const double mu_ang = sc.mu;
  cp_async_wait_all();
  __syncthreads();
  // the direct beam top * exp(tau / mu) of every level (photo.py:173-174), the
  // layers' optical depths, parked in the i_d row, and their albedos, in the phi row
  if (on) {
    const double top = P.sflux_top[bin], t_top = tb[(int64_t)nz * nbin];
    for (int j = row; j <= nz; j += PR) {
      const double t0 = j < nz ? iu[j * PB] : t_top;
      sb[j * PB] = top * exp(quot(t0, mu_ang));
      if (j < nz) id[j * PB] = t0 - (j + 1 < nz ? iu[(j + 1) * PB] : t_top);
    }
  }
  for (int j0 = row; j0 < nz && on; j0 += JL * PR) {
    double sa[JL], sT[JL], ss[JL];
    column_sums<PB, PR>(P, cs, wt, xT, nz, j0, bin, c, sa, sT, ss);
#pragma unroll
    for (int l = 0; l < JL; ++l) {
      const int j = j0 + l * PR;
      if (j < nz) {
        double tot_abs = 0.0, tot_scat = 0.0;
        if (P.n_abs > 0) tot_abs = sa[l];
        if (P.n_abs_T > 0) tot_abs = tot_abs + sT[l];
        if (P.n_scat > 0) tot_scat = ss[l];
        phi[j * PB] = albedo_of(tot_abs, tot_scat);
      }
    }
  }
  __syncthreads();
  if (on)
    for (int j = row; j < nz; j += PR) {
      const TwoStream q = two_stream(P, sc, phi[j * PB], id[j * PB]);
      const double dir0 = sb[j * PB] * (-mu_ang), dir1 = sb[(j + 1) * PB] * (-mu_ang);
      const double i_d = q.phi * q.gm * dir1 - (q.chi * q.gm + q.xi * q.gp) * dir0;
      const double i_u = q.phi * q.gp * dir0 - (q.xi * q.gm + q.chi * q.gp) * dir1;
      phi[j * PB] = q.phi;
      xi[j * PB] = q.xi;
      rc[j * PB] = 1.0 / q.chi;
      id[j * PB] = quot(i_d, mu_ang);
      iu[j * PB] = quot(i_u, mu_ang);
    }
  __syncthreads();
  if (threadIdx.x < PB && on) {
    // down recursion (photo.py:208-223) with dflux_u of the previous call, then
    // up (photo.py:225-236)
    // (a layer's chain is product, difference, sum and product; the operands of
    // four layers are loaded together, ahead of the four before)
    double v = 0.0;
    struct Four {
      double r[4], p[4], x[4], s[4];
    };
    // layers j, j + dir, ..: e walks the rows, all four inside the column
    auto load = [&](Four& o, int e, int dir, const double* w, const double* src) {
#pragma unroll
      for (int l = 0; l < 4; ++l, e += dir * PB) {
        o.r[l] = rc[e];
        o.p[l] = phi[e];
        o.x[l] = xi[e] * w[e];
        o.s[l] = src[e];
      }
    };
    auto chain = [&](const Four& o, double* out, int dir) {
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        v = o.r[l] * (o.p[l] * v - o.x[l] + o.s[l]);
        out[dir * l * PB] = v;
      }
    };
    // one direction: n layers from row e on, whole fours first
    auto sweep = [&](int e, int n, int dir, const double* w, const double* src, double* out) {
      Four a, c2;
      int left = n;
      if (left >= 4) load(a, e, dir, w, src);
#pragma unroll 1
      while (left >= 8) {
        load(c2, e + 4 * dir * PB, dir, w, src);
        chain(a, out + e, dir);
        e += 4 * dir * PB;
        left -= 4;
        if (left < 8) {
          a = c2;
          break;
        }
        load(a, e + 4 * dir * PB, dir, w, src);
        chain(c2, out + e, dir);
        e += 4 * dir * PB;
        left -= 4;
      }
      if (left >= 4) {
        chain(a, out + e, dir);
        e += 4 * dir * PB;
        left -= 4;
      }
      for (; left > 0; --left, e += dir * PB) {
        v = rc[e] * (phi[e] * v - xi[e] * w[e] + src[e]);
        out[e] = v;
      }
    };
    sweep((nz - 1) * PB, nz, -1, ud, id, ud);
    v = 0.0;
    sweep(0, nz - 1, 1, ud + PB, iu, id);   // level j + 1 into id[j]; the flux down into layer j from level j + 1
    const int e = (nz - 1) * PB;
    v = rc[e] * (phi[e] * v - xi[e] * 0.0 + iu[e]);
    id[e] = v;
  }
  __syncthreads();
  // actinic flux (photo.py:238-244) and the results of every level
  double change = 0.0;  // largest relative aflux change of this thread's entries above flux_atol
  if (on) {
    const double conv = P.hc / P.bins[bin];
    double* ab = aflux + (int64_t)b * nz * nbin + bin;
    for (int j = row; j <= nz; j += PR) {
      const double u_lo = j > 0 ? id[(j - 1) * PB] : 0.0, d_lo = j < nz ? ud[j * PB] : 0.0, s_lo = sb[j * PB];
      sflux[zb + (int64_t)j * nbin] = s_lo;
      dd[zb + (int64_t)j * nbin] = d_lo;
      du[zb + (int64_t)j * nbin] = u_lo;
      if (j < nz) {
        const double u_up = id[j * PB], d_up = j + 1 < nz ? ud[(j + 1) * PB] : 0.0, s_up = sb[(j + 1) * PB];
        const double ave = 0.5 * (s_lo + s_up);
        const double tot = ave + quot(0.5 * (u_lo + u_up + d_up + d_lo), P.edd);
        const double an = quot(tot, conv);
        if (achg && an > flux_atol) {
          const double r = fabs(an - ab[(int64_t)j * nbin]) / fmax(fabs(an), 1e-300);
          change = (r > change || r != r) ? r : change;
        }
        ab[(int64_t)j * nbin] = an;
      }
    }
  }
  // the ratios are >= 0 or NaN, so their bit patterns order as their values
  // do and a NaN wins the maximum, as it does in the reference's max
  if (achg) {
    unsigned long long m = static_cast<unsigned long long>(__double_as_longlong(change));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0 && m)
      atomicMax(reinterpret_cast<unsigned long long*>(achg + (int64_t)b * ACHG_STRIDE), m);
  }
}

__global__ void __launch_bounds__(PHOTO_THREADS)
flux_column_kernel(int nz, int ni, VbPhoto P, const double* __restrict__ tau, const double* __restrict__ ymix,
            const double* du_prev, double* __restrict__ aflux, double* __restrict__ sflux,
            double* __restrict__ dd, double* du, const int32_t* __restrict__ due, double flux_atol,
            double* __restrict__ achg) {
  // du_prev and du may be one buffer: each thread reads its bin of du_prev in
  // the down recursion before the up recursion overwrites it.
  const int b = blockIdx.y;
  const int bin = blockIdx.x * blockDim.x + threadIdx.x;
  if (due && due[b] == 0) return;
  if (bin >= P.nbin) return;
  const int nbin = P.nbin;
  const int64_t zb = (int64_t)b * (nz + 1) * nbin;
  const double* tb = tau + zb;
  const double* ym = ymix + (int64_t)b * nz * ni;
  const double* xT = P.absp_T_cross + (int64_t)b * P.T_stride;
  const double* up = du_prev + zb;
  double* sb = sflux + zb;
  double* ddb = dd + zb;
  double* dub = du + zb;
  double* ab = aflux + (int64_t)b * nz * nbin;
  const double mu_ang = -1.0 * P.mu_zenith;
  const double top = P.sflux_top[bin];
  // albedo of every layer, parked in the sflux rows until the up recursion
  // hands each row its direct beam (the sums over absorbers run once per
  // layer instead of once per recursion)
  for (int j = 0; j < nz; ++j) sb[(int64_t)j * nbin + bin] = albedo(P, xT, nz, ym + (int64_t)j * ni, j, bin);
  // down recursion (photo.py:208-223), dflux_u of the previous call; the
  // direct beam top * exp(tau / mu) (photo.py:173-174) level by level
  double d_next = 0.0;
  ddb[(int64_t)nz * nbin + bin] = 0.0;
  double s_hi = top * exp(tb[(int64_t)nz * nbin + bin] / mu_ang);
  for (int j = nz - 1; j >= 0; --j) {
    const double t0 = tb[(int64_t)j * nbin + bin], t1 = tb[(int64_t)(j + 1) * nbin + bin];
    const double s_lo = top * exp(t0 / mu_ang);
    TwoStream c = two_stream(P, StreamConst(P), sb[(int64_t)j * nbin + bin], t0 - t1);
    const double dir0 = s_lo * (-mu_ang);
    const double dir1 = s_hi * (-mu_ang);
    const double i_d = c.phi * c.gm * dir1 - (c.chi * c.gm + c.xi * c.gp) * dir0;
    const double v = (1.0 / c.chi) * (c.phi * d_next - c.xi * up[(int64_t)j * nbin + bin] + i_d / mu_ang);
    ddb[(int64_t)j * nbin + bin] = v;
    d_next = v;
    s_hi = s_lo;
  }
  // up recursion (photo.py:225-236) and the actinic flux (photo.py:238-244)
  double u_prev = 0.0;
  dub[bin] = 0.0;
  const double conv = P.hc / P.bins[bin];
  double change = 0.0;  // largest relative aflux change of this bin (entries above flux_atol)
  double s_lo = top * exp(tb[bin] / mu_ang);
  for (int j = 1; j <= nz; ++j) {
    const double t0 = tb[(int64_t)(j - 1) * nbin + bin], t1 = tb[(int64_t)j * nbin + bin];
    const double s_up = top * exp(t1 / mu_ang);
    TwoStream c = two_stream(P, StreamConst(P), sb[(int64_t)(j - 1) * nbin + bin], t0 - t1);
    const double dir0 = s_lo * (-mu_ang);
    const double dir1 = s_up * (-mu_ang);
    const double i_u = c.phi * c.gp * dir0 - (c.xi * c.gm + c.chi * c.gp) * dir1;
    const double v = (1.0 / c.chi) * (c.phi * u_prev - c.xi * ddb[(int64_t)j * nbin + bin] + i_u / mu_ang);
    dub[(int64_t)j * nbin + bin] = v;
    const double ave = 0.5 * (s_lo + s_up);
    const double tot = ave + 0.5 * (u_prev + v + ddb[(int64_t)j * nbin + bin] + ddb[(int64_t)(j - 1) * nbin + bin]) / P.edd;
    const double an = tot / conv;
    if (achg && an > flux_atol) {
      const double r = fabs(an - ab[(int64_t)(j - 1) * nbin + bin]) / fmax(fabs(an), 1e-300);
      change = (r > change || r != r) ? r : change;
    }
    ab[(int64_t)(j - 1) * nbin + bin] = an;
    sb[(int64_t)(j - 1) * nbin + bin] = s_lo;   // level j-1's albedo is spent: store its direct beam
    u_prev = v;
    s_lo = s_up;
  }
  sb[(int64_t)nz * nbin + bin] = s_lo;
  // the ratios are >= 0 or NaN, so their bit patterns order as their values
  // do and a NaN wins the maximum, as it does in the reference's max
  if (achg && change != 0.0)
    atomicMax(reinterpret_cast<unsigned long long*>(achg + (int64_t)b * ACHG_STRIDE),
              static_cast<unsigned long long>(__double_as_longlong(change)));
}

// J-rates of a tile of actinic-flux rows, all branches: JT layers of one
// atmosphere, or (ATM) one layer of JT due atmospheres that share the branch
// tables, so a temperature-dependent branch's row of that layer serves all of
// them as the others' rows serve every tile. The flux rows are staged once in
// shared memory and each warp takes up to JB branches at a time, so a staged
// flux value is read once per JB branches and a cross section once per tile (a
// small batch splits the branches over gridDim.z block groups). Lanes hold the
// partial sums, split at din12 for the two-resolution trapezoid
// (photo.py:316-349), then the k row (photo.py:465-478). With a branch at a time
// and tiles of layers, shared and L2 loads (two per product) bounded the
// kernel: 64 atmospheres, 120 layers, 2500 bins, 40 branches 640 us -> 272.
// A tile holds due atmospheres only (due_rows): a run whose atmospheres are due
// at different times would otherwise pay for four where one is due (update of 64
// atmospheres with 16 due 570 us -> 452, with all 1511 -> 1502).
constexpr int J_THREADS = 256;
constexpr int JW = J_THREADS / 32;
constexpr int J_ROWS = 4, J_BRANCHES = 5;   // of a full tile; a small batch takes single rows and branches

// The due atmospheres of ranks r0 .. r0 + JT - 1, by increasing index, into
// rows; returns how many there are (below 1: none). A thread takes a run of
// consecutive atmospheres; the block's prefix of the counts gives the ranks.
template <int JT>
__device__ inline int due_rows(const int32_t* __restrict__ due, int batch, int r0, int* rows) {
  __shared__ int sums[JW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (batch + J_THREADS - 1) / J_THREADS;
  const int a0 = min((int)threadIdx.x * per, batch), a1 = min(a0 + per, batch);
  int n = 0;
  for (int a = a0; a < a1; ++a) n += due[a] != 0;
  int incl = n;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += v;
  }
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  int rank = incl - n, total = 0;
#pragma unroll
  for (int q = 0; q < JW; ++q) {
    rank += q < warp ? sums[q] : 0;
    total += sums[q];
  }
  if (rank < r0 + JT && rank + n > r0)
    for (int a = a0; a < a1; ++a)
      if (due[a] != 0) {
        if (rank >= r0 && rank < r0 + JT) rows[rank - r0] = a;
        ++rank;
      }
  __syncthreads();
  return min(JT, total - r0);
}

template <bool ATM, int JT, int JB>
__global__ void __launch_bounds__(J_THREADS, 2)
j_kernel(int batch, int nz, int nr, int lt, VbPhoto P, const double* __restrict__ aflux, double* __restrict__ J_br,
         double* __restrict__ J_br_T, double* __restrict__ k, const int32_t* __restrict__ due) {
  extern __shared__ double fs[];   // [lt][nbin]
  __shared__ int rows[ATM ? JT : 1];   // the tile's atmospheres
  const int b0 = ATM ? blockIdx.y * lt : blockIdx.y, j0 = ATM ? blockIdx.x : blockIdx.x * lt;
  if (!ATM && due && due[b0] == 0) return;
  int nl = ATM ? min(lt, batch - b0) : min(lt, nz - j0);
  if (ATM && due) nl = due_rows<JT>(due, batch, b0, rows);
  if (nl <= 0) return;
  auto atm_of = [&](int l) { return !ATM ? b0 : due ? rows[l] : b0 + l; };
  auto layer_of = [&](int l) { return ATM ? j0 : j0 + l; };
  const int nbin = P.nbin, d12 = P.din12;
  for (int l = 0; l < nl; ++l) {
    const double* f = aflux + ((int64_t)atm_of(l) * nz + layer_of(l)) * nbin;
    for (int e = threadIdx.x; e < nbin; e += J_THREADS) fs[l * nbin + e] = f[e];
  }
  for (int e = nl * nbin + threadIdx.x; e < lt * nbin; e += J_THREADS) fs[e] = 0.0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nb = P.n_br + P.n_br_T, step = JW * gridDim.z;
  for (int br0 = blockIdx.z * JW + warp; br0 < nb; br0 += step * JB) {
    const double* c0[JB];
    int64_t cstep[JB];   // next flux row's cross sections (temperature-dependent branches of a layer tile)
#pragma unroll
    for (int u = 0; u < JB; ++u) {
      const int br = min(br0 + u * step, nb - 1);   // past the last branch: a repeat nobody reads
      const bool is_T = br >= P.n_br;
      // (a tile of atmospheres shares its tables: T_stride_J = 0)
      c0[u] = is_T ? P.cross_J_T + (ATM ? 0 : b0 * P.T_stride_J) + ((int64_t)(br - P.n_br) * nz + j0) * nbin
                   : P.cross_J + (int64_t)br * nbin;
      cstep[u] = is_T && !ATM ? nbin : 0;
    }
    double sum[2][JB][JT];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double(&s)[JB][JT] = sum[h];
#pragma unroll
      for (int u = 0; u < JB; ++u)
#pragma unroll
        for (int l = 0; l < JT; ++l) s[u][l] = 0.0;
      const int q1 = h == 0 ? d12 : nbin;
      for (int q = (h == 0 ? 0 : d12) + lane; q < q1; q += 32) {
        double f[JT];
#pragma unroll
        for (int l = 0; l < JT; ++l) f[l] = l < lt ? fs[l * nbin + q] : 0.0;
#pragma unroll
        for (int u = 0; u < JB; ++u) {
          if (ATM) {
            const double cv = c0[u][q];
#pragma unroll
            for (int l = 0; l < JT; ++l) s[u][l] = s[u][l] + f[l] * cv;
          } else {
#pragma unroll
            for (int l = 0; l < JT; ++l)
              if (l < nl) s[u][l] = s[u][l] + f[l] * c0[u][l * cstep[u] + q];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < JB; ++u)
#pragma unroll
        for (int l = 0; l < JT; ++l)
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) s[u][l] = s[u][l] + __shfl_xor_sync(0xffffffffu, s[u][l], off);
    }
    // lane u JT + l finishes branch u of row l
    double a1 = 0.0, a2 = 0.0;
#pragma unroll
    for (int u = 0; u < JB; ++u)
#pragma unroll
      for (int l = 0; l < JT; ++l)
        if (lane == u * JT + l) {
          a1 = sum[0][u][l];
          a2 = sum[1][u][l];
        }
    const int u = lane / JT, l = lane % JT, br = br0 + u * step;
    if (u < JB && l < nl && br < nb) {
      const bool is_T = br >= P.n_br;
      const int brl = is_T ? br - P.n_br : br, b = atm_of(l), j = layer_of(l);
      const double* f = fs + l * nbin;
      const double* c = is_T ? P.cross_J_T + (int64_t)b * P.T_stride_J + ((int64_t)brl * nz + j) * nbin
                             : P.cross_J + (int64_t)brl * nbin;
      double J = 0.0;
      if (d12 > 0) {
        double J1 = a1 * P.dbin1;
        J1 = J1 - 0.5 * (f[0] * c[0] + f[d12 - 1] * c[d12 - 1]) * P.dbin1;
        J = J1;
      }
      if (d12 < nbin) {
        double J2 = a2 * P.dbin2;
        J2 = J2 - 0.5 * (f[d12] * c[d12] + f[nbin - 1] * c[nbin - 1]) * P.dbin2;
        J = (d12 > 0) ? J + J2 : J2;
      }
      if (is_T) {
        if (J_br_T) J_br_T[((int64_t)b * P.n_br_T + brl) * nz + j] = J;
      } else {
        if (J_br) J_br[((int64_t)b * P.n_br + brl) * nz + j] = J;
      }
      if (k) {
        const int32_t* ridx = is_T ? P.br_T_re_idx : P.br_re_idx;
        const uint8_t* act = is_T ? P.br_T_active : P.br_active;
        if (ridx && act && act[brl]) k[((int64_t)b * (nr + 1) + ridx[brl]) * nz + j] = J * P.f_diurnal;
      }
    }
  }
}

static int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// Threads of a tile's CTA: 512 where one tile takes an SM's shared memory or
// the grid has no second one for it, else fewer, down to 128, until the tiles
// that an SM holds share its threads (sm_threads). With 512 for every tile a
// short column idles most of them (64 layers in flight) and the tiles of an SM
// run one after another. 2500 bins, 512 threads / this rule, us: flux of 64
// atmospheres of 20 layers 323 / 160, 43 layers 443 / 344, of 64 1233 / 980 at
// 126 (16 bins); tau of 64 of 20 layers 102 / 51, 90 layers 218 / 153.
static int tile_threads(size_t smem, int64_t tiles, int sms, int sm_threads) {
  const int64_t per_sm = std::min<int64_t>(227 * 1024 / (smem + 1024), (tiles + sms - 1) / sms);
  int t = 512;
  while (t > 128 && t * per_sm > sm_threads) t /= 2;
  return t;
}

// Whether a thread per bin and column is faster: a tile costs the same however
// short its column (a table of cross sections, five barriers, 16 layers a pass
// of 128 threads), a column's thread in proportion, so the line rises with the
// square of the layers. Flux, 2500 bins, us, tiles (128 threads) / columns: 2
// layers 4 atmospheres 7.5 / 10.5 and 8: 13.0 / 10.6, 4 layers 16: 21.0 / 18.9, 6
// layers 16: 24.8 / 27.2 and 32: 41.0 / 32.5, 8 layers 16: 26.5 / 34 and 64: 79 / 74,
// 10 layers 48: 71.7 / 67.1 and 128: 198 / 175, 14 layers 96: 171 / 176 and 256:
// 452 / 417, 18 layers 128: 297 / 311 and 256: 576 / 543, 20 layers 256: 602 / 615.
// Tau: 2 layers 8: 5.6 / 7.3 and 16: 9.6 / 7.4, 4 layers 16: 10.8 / 11.9 and 32:
// 16.3 / 12.3, 7 layers 48: 23.4 / 21.9, 8 layers 128: 54.9 / 53.0, 10 layers 256:
// 111 / 115.
static bool short_columns(int nz, int64_t tiles, int sms, bool flux) {
  const int64_t per_sm = flux ? std::max(nz + 2, nz * nz * (nz < 16 ? 5 : 6) / 20) : std::max(8, nz * nz / 2);
  return nz < (flux ? 20 : 10) && tiles >= sms * per_sm;
}

cudaError_t launch_photo_tau(int batch, int nz, int ni, const VbPhoto& P, const double* y, const double* dz,
                             double* tau, const int32_t* due, double* achg, cudaStream_t st) {
  constexpr int PB = 32;
  const size_t sm = tau_smem_bytes<PB>(P, nz);
  const dim3 grid((P.nbin + PB - 1) / PB, batch);
  const int64_t tiles = (int64_t)grid.x * batch;
  const int sms = sm_count();
  auto tiled = [&](auto kern, int threads) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    kern<<<grid, threads, sm, st>>>(nz, ni, P, y, dz, tau, due, achg);
    return cudaGetLastError();
  };
  if (sm <= PHOTO_SMEM_MAX && !short_columns(nz, tiles, sms, false)) {
    switch (tile_threads(sm, tiles, sms, 1024)) {
      case 128: return tiled(tau_kernel<PB, 128>, 128);
      case 256: return tiled(tau_kernel<PB, 256>, 256);
      default: return tiled(tau_kernel<PB, 512>, 512);
    }
  }
  dim3 grid1((P.nbin + PHOTO_THREADS - 1) / PHOTO_THREADS, batch);
  tau_column_kernel<<<grid1, PHOTO_THREADS, 0, st>>>(nz, ni, P, y, dz, tau, due, achg);
  return cudaGetLastError();
}

template <int PB>
static cudaError_t launch_flux_tiles(int batch, int nz, int ni, const VbPhoto& P, const double* tau,
                                     const double* ymix, const double* du_prev, double* aflux, double* sflux,
                                     double* dd, double* du, const int32_t* due, double flux_atol, double* achg,
                                     int sms, cudaStream_t st) {
  const size_t sm = flux_smem_bytes<PB>(P, nz);
  const dim3 grid((P.nbin + PB - 1) / PB, batch);
  auto launch = [&](auto kern, int threads) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    kern<<<grid, threads, sm, st>>>(nz, ni, P, tau, ymix, du_prev, aflux, sflux, dd, du, due, flux_atol, achg);
    return cudaGetLastError();
  };
  switch (tile_threads(sm, (int64_t)grid.x * batch, sms, FLUX_THREADS)) {
    case 128: return launch(flux_kernel<PB, 128>, 128);
    case 256: return launch(flux_kernel<PB, 256>, 256);
    default: return launch(flux_kernel<PB, 512>, 512);
  }
}

cudaError_t launch_photo_flux(int batch, int nz, int ni, const VbPhoto& P, const double* tau, const double* ymix,
                              const double* du_prev, double* aflux, double* sflux, double* dd, double* du,
                              const int32_t* due, double flux_atol, double* achg, cudaStream_t st) {
  const int species = P.n_abs + P.n_abs_T + P.n_scat, sms = sm_count();
  // 32 bins up to 120 layers or so, 16 up to 240
  if (!short_columns(nz, (int64_t)((P.nbin + 31) / 32) * batch, sms, true)) {
    if (species <= FLUX_MAX_SPECIES<32> && flux_smem_bytes<32>(P, nz) <= PHOTO_SMEM_MAX)
      return launch_flux_tiles<32>(batch, nz, ni, P, tau, ymix, du_prev, aflux, sflux, dd, du, due, flux_atol, achg,
                                   sms, st);
    if (species <= FLUX_MAX_SPECIES<16> && flux_smem_bytes<16>(P, nz) <= PHOTO_SMEM_MAX)
      return launch_flux_tiles<16>(batch, nz, ni, P, tau, ymix, du_prev, aflux, sflux, dd, du, due, flux_atol, achg,
                                   sms, st);
  }
  dim3 grid((P.nbin + PHOTO_THREADS - 1) / PHOTO_THREADS, batch);
  flux_column_kernel<<<grid, PHOTO_THREADS, 0, st>>>(nz, ni, P, tau, ymix, du_prev, aflux, sflux, dd, du, due,
                                                     flux_atol, achg);
  return cudaGetLastError();
}

cudaError_t launch_photo_j(int batch, int nz, int nr, const VbPhoto& P, const double* aflux, double* J_br,
                           double* J_br_T, double* k, const int32_t* due, cudaStream_t st) {
  if (P.n_br + P.n_br_T == 0) return cudaSuccess;
  // layers per block: JT when the batch fills the GPU with tiles, else one
  // layer per block (more blocks for a small batch); fewer when the flux rows
  // would not fit 200 KB of shared memory
  const int sms = sm_count();
  int lt = ((int64_t)batch * ((nz + J_ROWS - 1) / J_ROWS) >= 2 * (int64_t)sms) ? J_ROWS : 1;
  while (lt > 1 && (size_t)lt * P.nbin * sizeof(double) > 200 * 1024) --lt;
  if ((size_t)lt * P.nbin * sizeof(double) > 200 * 1024) return cudaErrorInvalidValue;
  const size_t smem = (size_t)lt * P.nbin * sizeof(double);
  // a batch that shares its tables tiles over atmospheres; a small batch also
  // spreads its branches over blocks (gridDim.z groups of JW)
  const bool by_atm = lt == J_ROWS && batch >= J_ROWS && P.T_stride_J == 0;
  const int groups = lt == 1 ? (P.n_br + P.n_br_T + JW - 1) / JW : 1;
  auto launch = [&](auto kern, dim3 grid) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<grid, J_THREADS, smem, st>>>(batch, nz, nr, lt, P, aflux, J_br, J_br_T, k, due);
    return cudaGetLastError();
  };
  if (by_atm) return launch(j_kernel<true, J_ROWS, J_BRANCHES>, dim3(nz, (batch + lt - 1) / lt, groups));
  const dim3 grid((nz + lt - 1) / lt, batch, groups);
  if (lt == 1) return launch(j_kernel<false, 1, 1>, grid);
  return launch(j_kernel<false, J_ROWS, J_BRANCHES>, grid);
}

}  // namespace vb
