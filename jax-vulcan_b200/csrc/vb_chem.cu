// Layer-parallel assembly kernels of the Ros2 step: chemistry RHS (mass-action
// rates gathered per species), analytic Jacobian (gathered per destination
// entry), eddy + molecular diffusion and boundary fluxes, fused into
//   * the stage-1 kernel: rhs(y) and the LHS blocks c0*I - J - diag(diff)
//     (reference jax_step.py:263-298, chem.py:83-214), and
//   * the stage-2 kernel: rhs(yk2) - 2/(r dt) k1 (jax_step.py:303-310).
// One CTA per layer, pair or tile of layers of an atmosphere. Compiled with
// --fmad=false: the gathers sum in the segment_sum order of the reference, so
// the RHS and the Jacobian are bit-identical to the reference's.
#include <cuda_runtime.h>

#include <algorithm>

#include "vb_common.cuh"
#include "vb_launch.cuh"
#include "vb_layer.cuh"

namespace vb {

struct LayerSmem {
  double* y3;      // [3][ni+1]: layers j-1, j, j+1 (padding slot = 1.0)
  double* diff;    // [ni]
  double* diagd;   // [ni]
  double* scal;    // [3]: ysum(j-1), ysum(j), ysum(j+1)
};

__host__ __device__ inline size_t layer_smem_bytes(int ni) {
  return (3 * (size_t)(ni + 1) + 2 * (size_t)ni + 3) * sizeof(double);
}

__device__ inline LayerSmem carve(double* s, int ni) {
  LayerSmem L;
  L.y3 = s; s += 3 * (ni + 1);
  L.diff = s; s += ni;
  L.diagd = s; s += ni;
  L.scal = s;
  return L;
}

// A reaction slot: its reactants' indices, the codes of their
// stoichiometries st[] (2 bits each; code 3: the value is read), and the
// three-body flag. One 8-byte word of a table that stays small in L1 for up to
// RX_TERMS terms; gathered from the wide tables above that.
struct Slot {
  uint64_t w;
  uint32_t codes;
  const int32_t* idx;
  const double* st;
  bool three;
};

template <int TT>
__device__ __forceinline__ Slot load_slot(const NetDev& net, int r) {
  Slot S;
  S.idx = net.r_idx + r * TT;
  S.st = net.r_st + r * TT;
  if (TT <= RX_TERMS) {
    S.w = __ldg(net.rx + r);
    S.codes = (uint32_t)(S.w >> 48);
    S.three = (S.w >> 60) & 1;
  } else {
    S.codes = 0;
#pragma unroll
    for (int s = 0; s < TT; ++s) S.codes |= st_code(S.st[s]) << (2 * s);
    S.three = net.three[r] != 0;
  }
  return S;
}

template <int TT>
__device__ __forceinline__ int slot_species(const Slot& S, int s) {
  return TT <= RX_TERMS ? (int)((S.w >> (8 * s)) & 0xff) : S.idx[s];
}

// Powers by code (pow_st's values): y**st (1 for a padding slot), and
// st y**(st-1), 0 unless st > 0.
struct WholePowers {
  template <int TT>
  __device__ __forceinline__ static double p(const Slot& S, int s, double y) {
    const uint32_t c = (S.codes >> (2 * s)) & 3u;
    return c == 0u ? 1.0 : c == 1u ? y : y * y;
  }
  template <int TT>
  __device__ __forceinline__ static double dp(const Slot& S, int s, double y) {
    const uint32_t c = (S.codes >> (2 * s)) & 3u;
    return c == 0u ? 0.0 : c == 1u ? 1.0 : 2.0 * y;
  }
};
struct AnyPowers {
  template <int TT>
  __device__ __forceinline__ static double p(const Slot& S, int s, double y) {
    return S.st[s] > 0.0 ? pow_st(y, S.st[s]) : 1.0;
  }
  template <int TT>
  __device__ __forceinline__ static double dp(const Slot& S, int s, double y) {
    return S.st[s] * (S.st[s] > 0.0 ? pow_st(y, S.st[s] - 1.0) : 0.0);
  }
};

// Rate of one reaction from its reactant values yr[] (padding slots st = 0),
// and with jac its derivative by each reactant slot into d[], in the
// reference's expression order (chem.py:92-99, 156-182). Shared by the
// per-layer and the layer-vectorized assembly.
template <int TT, class Powers>
__device__ __forceinline__ double rate_terms_p(const double (&yr)[TT], const Slot& S, double kr, double M, bool jac,
                                               double (&d)[TT]) {
  double f[TT];
#pragma unroll
  for (int s = 0; s < TT; ++s) f[s] = Powers::template p<TT>(S, s, yr[s]);
  double prod = f[0];
#pragma unroll
  for (int s = 1; s < TT; ++s) prod = prod * f[s];
  double rt = kr * prod;
  if (S.three) rt = rt * M;
  if (jac) {
#pragma unroll
    for (int s = 0; s < TT; ++s) {
      double lo = (s == 0) ? 1.0 : f[0];
#pragma unroll
      for (int t = 1; t < TT; ++t) lo = lo * ((t == s) ? 1.0 : f[t]);
      double dd = Powers::template dp<TT>(S, s, yr[s]);
      dd = dd * lo;
      dd = dd * kr;
      if (S.three) dd = dd * M;
      d[s] = dd;
    }
  }
  return rt;
}

// Whether a slot has a stoichiometry other than 0, 1 and 2.
template <int TT>
__device__ __forceinline__ bool any_powers(const Slot& S) {
  constexpr uint32_t LOW = 0x5555u & ((1u << (2 * TT)) - 1u);
  return (S.codes & (S.codes >> 1) & LOW) != 0;
}

// rate_terms_p of such a slot: out of line, so that pow takes neither
// registers nor instruction cache from the rest.
template <int TT>
__device__ __noinline__ double rate_terms_any(const double* y, const Slot& S, double kr, double M, bool jac,
                                              double* dout) {
  double yr[TT], d[TT];
#pragma unroll
  for (int s = 0; s < TT; ++s) yr[s] = y[s];
  const double rt = rate_terms_p<TT, AnyPowers>(yr, S, kr, M, jac, d);
  if (jac) {
#pragma unroll
    for (int s = 0; s < TT; ++s) dout[s] = d[s];
  }
  return rt;
}

// Values of NL layers at one index, interleaved in shared memory.
template <int NL>
struct Vals {
  double v[NL];
};
template <int NL>
__device__ __forceinline__ Vals<NL> ld_vals(const double* p, int i) {
  Vals<NL> r;
  if (NL == 2) {
    const double2 d = *reinterpret_cast<const double2*>(p + 2 * i);
    r.v[0] = d.x;
    r.v[NL - 1] = d.y;
  } else {
    r.v[0] = p[i];
  }
  return r;
}
template <int NL>
__device__ __forceinline__ void st_vals(double* p, int i, const double (&v)[NL]) {
  if (NL == 2)
    *reinterpret_cast<double2*>(p + 2 * i) = make_double2(v[0], v[NL - 1]);
  else
    p[i] = v[0];
}

// Rates (and drates) of reaction slot r with TT terms; yrow: the layers' state
// rows, ystride apart.
template <int TT, int NL, bool ANY>
__device__ inline void rate_slot(const Slot& S, int r, const double* yrow, int ystride, const double (&kr)[NL],
                                 const double (&M)[NL], double* rate, double* drate, bool jac) {
  double rt[NL], d[NL][TT];
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    double yr[TT];
#pragma unroll
    for (int s = 0; s < TT; ++s) yr[s] = yrow[l * ystride + slot_species<TT>(S, s)];
    if (ANY)
      rt[l] = rate_terms_any<TT>(yr, S, kr[l], M[l], jac, d[l]);
    else
      rt[l] = rate_terms_p<TT, WholePowers>(yr, S, kr[l], M[l], jac, d[l]);
  }
  st_vals<NL>(rate, r, rt);
  if (jac) {
#pragma unroll
    for (int s = 0; s < TT; ++s) {
      double v[NL];
#pragma unroll
      for (int l = 0; l < NL; ++l) v[l] = d[l][s];
      st_vals<NL>(drate, r * TT + s, v);
    }
  }
}

// Warps take blocks of 32 RU slots from a queue (zeroed before the barrier
// ahead of this), after the slots that need pow: one costs about 12,000 cycles
// (a long chain in code seldom in the instruction cache), which held up its
// warp's share and with it the layer. Rate constants of a block are loaded
// before any arithmetic so the strided L2 loads overlap (L2 only: the column
// of k would flush the gather tables from L1). kcol: the first layer's
// column; zs: the second's offset.
template <int TT, int NL, int RU>
__device__ inline void rates_t(const NetDev& net, const double* yrow, int ystride, const double* kcol,
                               int64_t kstride, int zs, const double (&M)[NL], int* queue, double* rate,
                               double* drate, bool jac) {
  const int lane = threadIdx.x & 31, n_any = (net.n_any + 31) / 32;
  while (true) {
    int q = 0;
    if (lane == 0) q = atomicAdd(queue, 1);
    q = __shfl_sync(0xffffffffu, q, 0);
    if (q < n_any) {
      if (32 * q + lane < net.n_any) {
        const int r = net.any_list[32 * q + lane];
        double kr[NL];
#pragma unroll
        for (int l = 0; l < NL; ++l) kr[l] = __ldcg(kcol + (int64_t)r * kstride + l * zs);
        rate_slot<TT, NL, true>(load_slot<TT>(net, r), r, yrow, ystride, kr, M, rate, drate, jac);
      }
      __syncwarp();
      continue;
    }
    const int r0 = 32 * RU * (q - n_any);
    if (r0 > net.nr) break;
    double kv[RU][NL];
    Slot S[RU];
#pragma unroll
    for (int u = 0; u < RU; ++u) {
      const int r = min(r0 + 32 * u + lane, net.nr);
#pragma unroll
      for (int l = 0; l < NL; ++l) kv[u][l] = __ldcg(kcol + (int64_t)r * kstride + l * zs);
      if (TT <= RX_TERMS) S[u] = load_slot<TT>(net, r);
    }
#pragma unroll
    for (int u = 0; u < RU; ++u) {
      const int r = r0 + 32 * u + lane;
      if (TT > RX_TERMS) S[u] = load_slot<TT>(net, min(r, net.nr));
      if (r <= net.nr && !any_powers<TT>(S[u]))
        rate_slot<TT, NL, false>(S[u], r, yrow, ystride, kv[u], M, rate, drate, jac);
    }
  }
}

// rate[r] = k[r] * prod_s y^st (* M) for every reaction slot of NL layers
// (chem.py:92-99); with jac, also drate[r][s] (chem.py:156-182).
template <int NL>
__device__ inline void layer_rates(const NetDev& net, const double* yrow, int ystride, const double* kcol,
                                   int64_t kstride, int zs, const double (&M)[NL], int* queue, double* rate,
                                   double* drate, bool jac) {
  constexpr int D = 3, DW = 2;
  if (!jac) {   // the right-hand-side kernels run at full occupancy: fewer loads in flight per thread
    switch (net.T) {
      case 1: rates_t<1, NL, 2>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
      case 2: rates_t<2, NL, 2>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
      case 3: rates_t<3, NL, 2>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
      case 4: rates_t<4, NL, 2>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
      case 5: rates_t<5, NL, 2>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
      case 6: rates_t<6, NL, 2>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
      case 7: rates_t<7, NL, 2>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
      default: rates_t<8, NL, 2>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
    }
  }
  switch (net.T) {
    case 1: rates_t<1, NL, D>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
    case 2: rates_t<2, NL, D>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
    case 3: rates_t<3, NL, D>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
    case 4: rates_t<4, NL, D>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
    case 5: rates_t<5, NL, DW>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
    case 6: rates_t<6, NL, DW>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
    case 7: rates_t<7, NL, DW>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
    default: rates_t<8, NL, DW>(net, yrow, ystride, kcol, kstride, zs, M, queue, rate, drate, jac); return;
  }
}

// The coefficient table of the gathers into shared memory (coef[MAX_COEF + 1]).
__device__ inline void load_coefs(const NetDev& net, double* coef) {
  if (net.coef_packed) return;
  for (int c = threadIdx.x; c < net.n_coef; c += blockDim.x) coef[c] = net.coef_tab[c];
}

// Coefficient of a term word: its own upper half (PK) or the table's entry.
template <bool PK>
__device__ __forceinline__ double term_coef(const double* coef, uint32_t x) {
  return PK ? __hiloint2double((int)(x & 0xffff0000u), 0) : coef[x >> 16];
}

constexpr int GW = 8;   // term words of a list held ahead by a lane

// Words k .. of a group (wp: the lane's first word) that exist.
__device__ __forceinline__ void group_words(const uint32_t* wp, int len, uint32_t (&w)[GW]) {
#pragma unroll
  for (int u = 0; u < GW; ++u) w[u] = u < len ? __ldg(wp + 32 * u) : 0u;
}

// Sums of a lane's list of cnt terms, in list order; len: the group's longest.
// w holds the first GW words; each half is reloaded GW terms ahead as it is used.
// load(i): the values at index i.
template <bool PK, int NL, typename Load>
__device__ __forceinline__ void gather_list(const double* coef, Load load, const uint32_t* wp, int len, int cnt,
                                            uint32_t (&w)[GW], double (&acc)[NL]) {
  constexpr int H = GW / 2;
#pragma unroll
  for (int l = 0; l < NL; ++l) acc[l] = 0.0;
  for (int k = 0; k < len; k += GW) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k0 = k + h * H;
      if (k0 >= len) break;
      Vals<NL> v[H];
      double c[H];
#pragma unroll
      for (int u = 0; u < H; ++u) {
        v[u] = load((int)(w[h * H + u] & 0xffffu));
        c[u] = term_coef<PK>(coef, w[h * H + u]);
      }
#pragma unroll
      for (int u = 0; u < H; ++u) w[h * H + u] = k0 + GW + u < len ? __ldg(wp + 32 * (k0 + GW + u)) : 0u;
#pragma unroll
      for (int u = 0; u < H; ++u) {
#pragma unroll
        for (int l = 0; l < NL; ++l) {
          const double t = acc[l] + c[u] * v[u].v[l];
          if (k0 + u < cnt) acc[l] = t;
        }
      }
    }
  }
}

// A long group's lane sums.
template <bool PK, int NL>
__device__ __forceinline__ void gather_group(const NetDev& net, const double* coef, const double* src, int g,
                                             uint32_t desc, double (&acc)[NL]) {
  const uint32_t b0 = net.gl_base[g], b1 = net.gl_base[g + 1];
  const int len = (int)(b1 - b0) / 32;
  const uint32_t* wp = net.gl_w + b0 + (threadIdx.x & 31);
  uint32_t w[GW];
  group_words(wp, len, w);
  gather_list<PK, NL>(coef, [&](int i) { return ld_vals<NL>(src, i); }, wp, len, (int)(desc & 0xffffu), w, acc);
}

// Up to GB groups of short entries, from group g (n of them exist): all words
// first, so the table's latency is paid once. Every list has GL_SHORT words,
// though three quarters of the entries have fewer terms: without classes by
// length the entries stay in storage order, and a warp's store touches 9
// sectors, not 27. Measured on B200 (stage 1 with the diffusion rows, 296
// atmospheres of 69 species, two layers per CTA / 128 of 89 species): a class
// per length 2.08 / 1.94 ms, lists filled up to 2 or 4 terms 1.97 / 1.79, to 4
// 1.97 / 1.76, to 3 or 8 2.05 / 1.75. Ordering the lists of equal length so
// that a quarter-warp's reads share fewer banks, at the cost of the stores'
// order, was slower (2.14 / 2.08).
constexpr int GB = 4;
template <bool PK, int NL, typename Off>
__device__ __forceinline__ void gather_short(const NetDev& net, const double* coef, const double* drate, int g, int n,
                                             Off off) {
  constexpr int C = GL_SHORT;
  const int lane = threadIdx.x & 31;
  const uint32_t* wp = net.gl_w + net.gl_base[g] + lane;
  uint32_t desc[GB], w[GB][C];
#pragma unroll
  for (int q = 0; q < GB; ++q) {
    desc[q] = q < n ? __ldg(net.gl_desc + 32 * (g + q) + lane) : ~0u;
#pragma unroll
    for (int u = 0; u < C; ++u) w[q][u] = q < n ? __ldg(wp + 32 * (C * q + u)) : 0u;
  }
#pragma unroll
  for (int q = 0; q < GB; ++q) {
    double J[NL];
#pragma unroll
    for (int l = 0; l < NL; ++l) J[l] = 0.0;
#pragma unroll
    for (int u = 0; u < C; ++u) {
      const double c = term_coef<PK>(coef, w[q][u]);
      const Vals<NL> v = ld_vals<NL>(drate, (int)(w[q][u] & 0xffffu));
#pragma unroll
      for (int l = 0; l < NL; ++l) J[l] = J[l] + c * v.v[l];
    }
    if (desc[q] != ~0u) off((int)((desc[q] >> 16) & 0x7fu), (int)(desc[q] >> 23), J);
  }
}

// The gathers of NL layers: the species lists' sums to part[t] (sums), the
// Jacobian's diagonal entries to diag(row, J), the others to off(row, col, J),
// each in the reference's order. The warps take work from a queue in shared
// memory (zeroed before the barrier ahead of this), the long groups first and
// one by one, then the short ones GB at a time, so they finish together. What
// bounds this is instructions issued and shared-memory wavefronts, not the
// latency of the tables: hence code without counts for the short lists, the
// diagonal's extra terms out of the common path, and the coefficient in the
// word. drate[(nr+1)*T] of each layer is 0 (fillers of short lists).
template <bool PK, int NL, typename Diag, typename Off>
__device__ __forceinline__ void gather_layer_t(const NetDev& net, const double* coef, const double* rate,
                                               const double* drate, bool sums, int* queue, double* part, Diag diag,
                                               Off off) {
  const int lane = threadIdx.x & 31;
  const int g0 = sums ? 0 : net.gl_sums;
  while (true) {
    int g = 0;
    if (lane == 0) g = atomicAdd(queue, 1);
    g = g0 + __shfl_sync(0xffffffffu, g, 0);
    if (g < net.gl_long) {
      const uint32_t desc = net.gl_desc[32 * g + lane];
      const bool on = desc != ~0u;
      double acc[NL];
      gather_group<PK, NL>(net, coef, g < net.gl_sums ? rate : drate, g, on ? desc : 0u, acc);
      if (!on) continue;
      const int row = (int)((desc >> 16) & 0x7fu);
      if (g < net.gl_sums)
        st_vals<NL>(part, (int)(desc >> 16), acc);
      else if (g < net.gl_diag)
        diag(row, acc);
      else
        off(row, (int)(desc >> 23), acc);
      continue;
    }
    g = net.gl_long + GB * (g - net.gl_long);
    if (g >= net.gl_groups) break;
    gather_short<PK, NL>(net, coef, drate, g, net.gl_groups - g, off);
  }
}

template <int NL, typename Diag, typename Off>
__device__ __forceinline__ void gather_layer(const NetDev& net, const double* coef, const double* rate,
                                             const double* drate, bool sums, int* queue, double* part, Diag diag,
                                             Off off) {
  if (net.coef_packed)
    gather_layer_t<true, NL>(net, coef, rate, drate, sums, queue, part, diag, off);
  else
    gather_layer_t<false, NL>(net, coef, rate, drate, sums, queue, part, diag, off);
}

// Loss and production sums of every species: part[2i] = loss_i, part[2i+1] =
// prod_i. The caller synchronises before reading dy_i/dt = part[2i+1] - part[2i].
template <bool PK, int NL>
__device__ __forceinline__ void species_sums_t(const NetDev& net, const double* coef, const double* rate,
                                               double* part) {
  for (int g = (int)threadIdx.x / 32; g < net.gl_sums; g += (int)blockDim.x / 32) {
    const uint32_t desc = net.gl_desc[32 * g + (threadIdx.x & 31)];
    double acc[NL];
    gather_group<PK, NL>(net, coef, rate, g, desc == ~0u ? 0u : desc, acc);
    if (desc != ~0u) st_vals<NL>(part, (int)(desc >> 16), acc);
  }
}

template <int NL>
__device__ inline void species_sums(const NetDev& net, const double* coef, const double* rate, double* part) {
  if (net.coef_packed)
    species_sums_t<true, NL>(net, coef, rate, part);
  else
    species_sums_t<false, NL>(net, coef, rate, part);
}

// Loads state rows j-1..j+1 and their gas sums.
__device__ inline void load_rows(const double* y, const double* gas, int nz, int ni, int j, LayerSmem& L) {
  for (int t = threadIdx.x; t < 3 * (ni + 1); t += blockDim.x) {
    int w = t / (ni + 1), i = t % (ni + 1);
    int jj = j - 1 + w;
    double v = 1.0;
    if (i < ni) v = (jj >= 0 && jj < nz) ? y[(int64_t)jj * ni + i] : 0.0;
    L.y3[t] = v;
  }
  // the gas mask staged in diagd (free until the diffusion writes it), so the
  // three sums below read shared memory
  for (int i = threadIdx.x; i < ni; i += blockDim.x) L.diagd[i] = gas[i];
  __syncthreads();
  if (threadIdx.x < 3) {
    int w = threadIdx.x;
    int jj = j - 1 + w;
    double s = 0.0;
    if (jj >= 0 && jj < nz) s = pairwise_sum_masked(L.y3 + w * (ni + 1), L.diagd, ni);
    L.scal[w] = s;
  }
  __syncthreads();
}

// Diffusion term of species i on row j from its combined coefficients and
// state values y(j), y(j-1), y(j+1): the stencil and the boundary fluxes
// (jax_step.py:223-246, _apply_diffusion_jax).
__device__ inline double diffusion_term(const AtmRef& a, int nz, int j, int i, int flags, double At, double Bt,
                                        double Ct, double y0, double ym, double yp) {
  double d;
  if (j == 0) {
    d = At * y0 + Bt * yp;
  } else if (j == nz - 1) {
    d = At * y0 + Ct * ym;
  } else {
    d = At * y0 + Bt * yp + Ct * ym;
  }
  if (j == nz - 1) {
    d = d + ((flags & VB_USE_TOPFLUX) ? a.top[i] / a.dzi[nz - 2] : 0.0);
  }
  if (j == 0) {
    d = d + ((flags & VB_USE_BOTFLUX) ? (a.bot[i] - y0 * a.vdep[i]) / a.dzi[0] : 0.0);
  }
  return d;
}

// diff[i] (with BC fluxes) and the diagonal diffusion term diag_d[i] of row j;
// also the sup/sub coefficients of row j when requested.
__device__ inline void layer_diffusion(const AtmRef& a, int nz, int ni, int j, int flags, LayerSmem& L,
                                       double* sup_out, double* sub_out) {
  double ysm = L.scal[0], ys0 = L.scal[1], ysp = L.scal[2];
  __shared__ double eddy[3];
  if (threadIdx.x == 0) {
    double A, B, C;
    eddy_row(a, nz, j, ysm, ys0, ysp, A, B, C);
    eddy[0] = A; eddy[1] = B; eddy[2] = C;
  }
  __syncthreads();
  double use_vm = (flags & VB_USE_VM_MOL) ? 1.0 : 0.0;
  double use_set = (flags & VB_USE_SETTLING) ? 1.0 : 0.0;
  const double* y0 = L.y3 + (ni + 1);
  const double* ym = L.y3;
  const double* yp = L.y3 + 2 * (ni + 1);
  for (int i = threadIdx.x; i < ni; i += blockDim.x) {
    double Am, Bm, Cm;
    mol_row(a, nz, ni, j, i, ysm, ys0, ysp, use_vm, use_set, Am, Bm, Cm);
    double At = eddy[0] + Am;
    double Bt = eddy[1] + Bm;
    double Ct = eddy[2] + Cm;
    L.diff[i] = diffusion_term(a, nz, j, i, flags, At, Bt, Ct, y0[i], ym[i], yp[i]);
    L.diagd[i] = At;
    if (sup_out && j < nz - 1) sup_out[i] = Bt;
    if (sub_out && j > 0) sub_out[i] = Ct;
  }
}

// Shared memory of stage1_kernel<NL>: the drates (and a 0) and rates of NL
// layers interleaved (16-byte aligned at NL = 2), then sums, rows and diagonals.
__host__ __device__ inline size_t stage1_smem_bytes(int ni, int nr, int T, int NL) {
  return (size_t)NL * ((size_t)(nr + 1) * (T + 1) + 1 + 2 * (size_t)ni + (ni + 1) + ni) * sizeof(double);
}

// Stage-1 assembly: rmod[j] = rhs(y), inv[j] = c0*I - J - diag(diag_d),
// supn[j] = -sup_d, subn[j-1] = -sub_d, with fix_mask (jax_step.py:263-298),
// of layers j0 .. j0 + NL - 1, j0 = NL blockIdx.x.
// Measured on B200, ni=69, nr=1400, nz=120, 296 atmospheres, with the diffusion
// rows, one layer per CTA, four CTAs per SM (the shared-memory limit): 2.71 ms
// with the lists dealt out in fixed bands, coefficients in a table and pow in
// line (681 M instructions in a ragged batch of 85, issue slots 70 % busy);
// 2.92 with the queue alone; 2.46 with code without counts for the short lists
// and packed reaction words (406 M); 2.35 with pow out of line; 2.02 with the
// short entries in storage order; 1.98 with two layers per CTA, where 512
// threads beat 384 (2.20 against 2.07 at that point) and 256 (2.44); 1.86 with
// the rows kernel's zero numerators; 1.78 with the slots that need pow ahead of
// the others. What is left is the wavefronts of the scattered shared-memory reads.
template <int NL>
__global__ void __launch_bounds__(NL * LAYER_THREADS, 4 / NL)
stage1_kernel(NetDev net, Batch B, const double* __restrict__ y, const double* __restrict__ k,
              const double* __restrict__ dt, const double* __restrict__ atm, int flags,
              const uint8_t* __restrict__ fix_mask, double* __restrict__ ws, const double* __restrict__ adj_v) {
  extern __shared__ __align__(16) double smem[];
  const int b = blockIdx.y, j = NL * blockIdx.x;
  Geo g = geo_of(B, b);
  if (j >= g.nz) return;
  const int ni = B.ni, nz = g.nz, ld = B.ld;
  const int nl = min(NL, nz - j);                 // layers here
  const int last = nl - 1;                        // a missing layer repeats the last, without stores
  double* drate = smem;                           // [(nr+1)*T + 1][NL]
  double* rate = drate + NL * ((B.nr + 1) * net.T + 1);   // [nr+1][NL]
  double* part = rate + NL * (B.nr + 1);          // [2 ni][NL]
  double* yj = part + NL * 2 * ni;                // [NL][ni+1]
  double* diagd = yj + NL * (ni + 1);             // [NL][ni]
  AtmRef a = atm_ref(atm + g.atm, nz, ni);
  WsView w = ws_view(ws, g, ni, ld);
  const double* yb = y + g.z0 * ni;
  const uint8_t* fm = fix_mask ? fix_mask + g.z0 * ni + (int64_t)j * ni : nullptr;
  const bool adj = adj_v != nullptr;   // J_y blocks of the steady-state adjoint
  const double r = ros2_r();
  const double c0 = adj ? 0.0 : 1.0 / (r * dt[b]);

  __shared__ double coefs[MAX_COEF + 1];
  __shared__ int queue, slots;
  if (threadIdx.x == 0) queue = slots = 0;
  if (threadIdx.x < NL) drate[NL * (B.nr + 1) * net.T + threadIdx.x] = 0.0;
  load_coefs(net, coefs);
  // state rows (the rates; padding slot 1.0) and diag_d, written with the rows'
  // diffusion terms by diffusion_rows_kernel ahead of this kernel
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    const int64_t q = (int64_t)(j + min(l, last)) * ni;
    for (int t = threadIdx.x; t <= ni; t += blockDim.x) yj[l * (ni + 1) + t] = t < ni ? yb[q + t] : 1.0;
    for (int i = threadIdx.x; i < ni; i += blockDim.x) diagd[l * ni + i] = w.aux[q + i];
  }
  __syncthreads();
  double M[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) M[l] = a.M[j + min(l, last)];
  layer_rates<NL>(net, yj, ni + 1, k + g.z0 * (B.nr + 1) + j, nz, last, M, &slots, rate, drate, true);
  __syncthreads();
  // One phase for the species sums and the Jacobian gather. The gather writes
  // each block entry in its final form.
  double* blk = w.inv + (int64_t)j * ni * ld;
  const int64_t lstep = (int64_t)ni * ld;
  const double bot = (j == 0 && (flags & VB_USE_BOTFLUX)) ? 1.0 : 0.0;
  auto depth = [&](int row, int l) { return l == 0 && j == 0 ? (bot != 0.0 ? -a.vdep[row] / a.dzi[0] : 0.0) : 0.0; };
  if (adj) {
    // steady_state_grad.py:153-175: diag = J + diag(A_eddy + A_mol) (+ deposition
    // at the bottom), sup_d = B[:-1], sub_d = C[1:] (no c0, not negated); no sums
    gather_layer<NL>(
        net, coefs, rate, drate, false, &queue, part,
        [&](int row, const double (&J)[NL]) {
#pragma unroll
          for (int l = 0; l < NL; ++l) {
            double v = J[l] + diagd[l * ni + row];
            if (l == 0 && j == 0) v = v + depth(row, l);
            if (l < nl) blk[l * lstep + (int64_t)row * ld + row] = v;
          }
        },
        [&](int row, int col, const double (&J)[NL]) {
#pragma unroll
          for (int l = 0; l < NL; ++l)
            if (l < nl) blk[l * lstep + (int64_t)row * ld + col] = J[l];
        });
    for (int i = threadIdx.x; i < nl * ni; i += blockDim.x)
      w.rmod[(int64_t)j * ni + i] = adj_v[g.z0 * ni + (int64_t)j * ni + i];
    return;
  }
  gather_layer<NL>(
      net, coefs, rate, drate, true, &queue, part,
      [&](int row, const double (&J)[NL]) {
#pragma unroll
        for (int l = 0; l < NL; ++l) {
          double v = c0 - J[l];
          // jax_step.py:283,288: the deposition term joins diag_d before -diag_d is added
          double dd = diagd[l * ni + row];
          if (l == 0 && j == 0) dd = dd + depth(row, l);
          v = v + (-dd);
          if (l < nl) {
            if (fm && fm[l * ni + row]) v = c0;
            blk[l * lstep + (int64_t)row * ld + row] = v;
          }
        }
      },
      [&](int row, int col, const double (&J)[NL]) {
#pragma unroll
        for (int l = 0; l < NL; ++l) {
          if (l < nl) {
            double v = 0.0 - J[l];
            if (fm && fm[l * ni + row]) v = 0.0;
            blk[l * lstep + (int64_t)row * ld + col] = v;
          }
        }
      });
  __syncthreads();   // the species sums
  for (int t = threadIdx.x; t < nl * ni; t += blockDim.x) {
    const int l = t >= ni ? 1 : 0, i = t - l * ni;
    // rmod[j] holds the row's diffusion term (diffusion_rows_kernel)
    double v = (part[NL * (2 * i + 1) + l] - part[NL * 2 * i + l]) + w.rmod[(int64_t)j * ni + t];
    if (fm && fm[t]) v = 0.0;
    w.rmod[(int64_t)j * ni + t] = v;
  }
}

__host__ __device__ inline size_t stage2_smem_bytes(int ni, int nr, int NL) {
  return (size_t)NL * ((size_t)(nr + 1) + 2 * (size_t)ni + (ni + 1)) * sizeof(double);
}

// Stage-2 right-hand side: rmod[j] = rhs(yk2) - 2/(r dt) k1[j] with
// yk2 = y + k1/r (jax_step.py:303-310), of layers j .. j + NL - 1. No drate
// buffer, so eight CTAs of one layer fit an SM; occupancy, not per-thread ILP,
// hides the gathers' latency (measured on B200, ni=69, nr=1400, 296
// atmospheres: 3 / 4 / 5 / 6 CTAs per SM 2.22 / 1.87 / 1.70 / 1.57 ms; 8 with
// rate constants loaded 2 deep instead of 6: 1.53 ms, despite the spills at 32
// registers).
template <int NL>
__global__ void __launch_bounds__(NL * LAYER_THREADS, 8 / NL)
stage2_kernel(NetDev net, Batch B, const double* __restrict__ y, const double* __restrict__ k,
              const double* __restrict__ dt, const double* __restrict__ atm,
              const uint8_t* __restrict__ fix_mask, double* __restrict__ ws, double* __restrict__ resid) {
  extern __shared__ __align__(16) double smem[];
  const int b = blockIdx.y, j = NL * blockIdx.x;
  Geo g = geo_of(B, b);
  if (j >= g.nz) return;
  const int ni = B.ni, nz = g.nz;
  const int nl = min(NL, nz - j), last = nl - 1;   // layers here; a missing one repeats the last
  double* rate = smem;                        // [nr+1][NL]
  double* part = rate + NL * (B.nr + 1);      // [2 ni][NL]
  double* yj = part + NL * 2 * ni;            // [NL][ni+1]
  AtmRef a = atm_ref(atm + g.atm, nz, ni);
  WsView w = ws_view(ws, g, ni, B.ld);
  const double* yb = y + g.z0 * ni;
  const uint8_t* fm = fix_mask ? fix_mask + g.z0 * ni + (int64_t)j * ni : nullptr;
  const double r = ros2_r();
  const bool res = resid != nullptr;   // steady-state residual f(y) (steady_state_grad.py:116-130)
  const double dtb = res ? 1.0 : dt[b];

  __shared__ double coefs[MAX_COEF + 1];
  __shared__ int slots;
  if (threadIdx.x == 0) slots = 0;
  load_coefs(net, coefs);
  // state rows (yk2 = y + k1/r; padding slot 1.0)
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    const int64_t q = (int64_t)(j + min(l, last)) * ni;
    for (int t = threadIdx.x; t <= ni; t += blockDim.x) {
      double v = 1.0;
      if (t < ni) {
        v = yb[q + t];
        if (!res) v = v + w.k1[q + t] / r;
      }
      yj[l * (ni + 1) + t] = v;
    }
  }
  __syncthreads();
  double M[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) M[l] = a.M[j + min(l, last)];
  layer_rates<NL>(net, yj, ni + 1, k + g.z0 * (B.nr + 1) + j, nz, last, M, &slots, rate, nullptr, false);
  __syncthreads();
  species_sums<NL>(net, coefs, rate, part);
  __syncthreads();
  // rmod[j] (resid[j]) holds the row's diffusion term (diffusion_rows_kernel)
  const double* dif = res ? resid + g.z0 * ni : w.rmod;
  for (int t = threadIdx.x; t < nl * ni; t += blockDim.x) {
    const int l = t >= ni ? 1 : 0, i = t - l * ni;
    const int64_t q = (int64_t)j * ni + t;
    double v = (part[NL * (2 * i + 1) + l] - part[NL * 2 * i + l]) + dif[q];
    if (res) {
      resid[g.z0 * ni + q] = v;
      continue;
    }
    if (fm && fm[t]) v = 0.0;
    w.rmod[q] = v - (2.0 / (r * dtb)) * w.k1[q];
  }
}

// Standalone chemistry: dydt (and optionally the Jacobian) of a uniform batch.
__host__ __device__ inline size_t chem_smem_bytes(int ni, int nr, int T, bool jac) {
  return ((size_t)(nr + 1) + 2 * (size_t)ni + (ni + 1) + (jac ? (size_t)(nr + 1) * T + 1 + (size_t)ni * ni : 0)) *
         sizeof(double);
}

// The right-hand side has a kernel of its own: with the Jacobian's registers two
// CTAs fit an SM, and a layer of a small network is one round of dependent
// loads, which only other CTAs hide. Right-hand side of 60 layers (B200, us, one
// kernel for both / four / six / eight CTAs per SM): 64 atmospheres of 12 species
// 63 / 35 / 28 / 29, 200 of 30: 232 / 127 / 103 / 114, 64 of 89: 110 / 82 / 65 / 68,
// one of 69: 9.1 / 8.7 / 8.8 / 10.0.
template <bool JAC>
__global__ void __launch_bounds__(LAYER_THREADS, JAC ? 2 : 6)
chem_kernel(NetDev net, int nz, const double* __restrict__ y, const double* __restrict__ M,
            const double* __restrict__ k, double* __restrict__ dydt, double* __restrict__ jac) {
  extern __shared__ __align__(16) double smem[];
  const int b = blockIdx.y, j = blockIdx.x;
  const int ni = net.ni;
  double* rate = smem;                            // [nr+1]
  double* part = rate + (net.nr + 1);             // [2 ni]
  double* yj = part + 2 * ni;                     // [ni+1]
  double* drate = yj + (ni + 1);                  // [(nr+1)*T + 1]
  double* J = drate + (net.nr + 1) * net.T + 1;   // [ni][ni]
  const double* yrow = y + ((int64_t)b * nz + j) * ni;
  __shared__ double coefs[MAX_COEF + 1];
  __shared__ int queue, slots;
  if (threadIdx.x == 0) {
    queue = slots = 0;
    if (JAC) drate[(net.nr + 1) * net.T] = 0.0;
  }
  load_coefs(net, coefs);
  for (int i = threadIdx.x; i <= ni; i += blockDim.x) yj[i] = i < ni ? yrow[i] : 1.0;
  __syncthreads();
  const double Mj[1] = {M[(int64_t)b * nz + j]};
  layer_rates<1>(net, yj, 0, k + (int64_t)b * (net.nr + 1) * nz + j, nz, 0, Mj, &slots, rate, drate, JAC);
  __syncthreads();
  if (JAC)
    gather_layer<1>(
        net, coefs, rate, drate, true, &queue, part, [&](int row, const double (&v)[1]) { J[row * ni + row] = v[0]; },
        [&](int row, int col, const double (&v)[1]) { J[row * ni + col] = v[0]; });
  else
    species_sums<1>(net, coefs, rate, part);
  __syncthreads();
  if (dydt)
    for (int i = threadIdx.x; i < ni; i += blockDim.x)
      dydt[((int64_t)b * nz + j) * ni + i] = part[2 * i + 1] - part[2 * i];
  if (JAC) {
    double* out = jac + ((int64_t)b * nz + j) * ni * ni;
    for (int d = threadIdx.x; d < ni * ni; d += blockDim.x) out[d] = J[d];
  }
}

// Standalone diffusion of a uniform batch (jax_step.py:67-246).
__global__ void __launch_bounds__(LAYER_THREADS)
diffusion_kernel(int nz, int ni, const double* __restrict__ y, const double* __restrict__ atm,
                 int flags, double* __restrict__ diff, double* __restrict__ diag_d,
                 double* __restrict__ sup_d, double* __restrict__ sub_d) {
  extern __shared__ __align__(16) double smem[];
  const int b = blockIdx.y, j = blockIdx.x;
  LayerSmem L = carve(smem, ni);
  AtmRef a = atm_ref(atm + (int64_t)b * VB_ATM_DOUBLES(nz, ni), nz, ni);
  const double* yb = y + (int64_t)b * nz * ni;
  load_rows(yb, a.gas, nz, ni, j, L);
  __syncthreads();
  double* supo = sup_d ? sup_d + ((int64_t)b * (nz - 1) + j) * ni : nullptr;
  double* subo = sub_d ? sub_d + ((int64_t)b * (nz - 1) + (j - 1)) * ni : nullptr;
  layer_diffusion(a, nz, ni, j, flags, L, supo, subo);
  __syncthreads();
  for (int i = threadIdx.x; i < ni; i += blockDim.x) {
    if (diff) diff[((int64_t)b * nz + j) * ni + i] = L.diff[i];
    if (diag_d) {
      double dd = L.diagd[i];
      if (j == 0) dd = dd + ((flags & VB_USE_BOTFLUX) ? -a.vdep[i] / a.dzi[0] : 0.0);
      diag_d[((int64_t)b * nz + j) * ni + i] = dd;
    }
  }
}

// ---------------------------------------------------------------- diffusion rows ahead of the stages
// The eddy + molecular diffusion of every layer (the same functions on the
// same inputs as layer_diffusion, so the same bits), computed ahead of the
// stage kernels, whose heavy per-layer CTAs then load one state row and no
// atmosphere fields. One CTA per block of DIFF_LAYERS consecutive layers of
// one atmosphere: the block's state rows, their gas sums, per-layer fields
// and eddy coefficients are formed once, then every (layer, species) item of
// the block runs in parallel.
//   mode 0 (stage 1):  rmod[j] = diff, aux[j] = diag_d, supn[j] = -sup_d,
//                      subn[j-1] = -sub_d (0 on fixed species);
//   mode 1 (stage 1 of the adjoint): aux[j] = diag_d, supn[j] = sup_d,
//                      subn[j-1] = sub_d (steady_state_grad.py:153-175);
//   mode 2 (stage 2):  rmod[j] = diff at yk2 = y + k1/r (with resid: resid[j]
//                      = diff at y, the residual; ws unused).
// Four CTAs per SM (64 registers, 32 bytes spilled): 0.239 ms per launch, before
// zero numerators were kept out of the divisions (0.117 since), at
// 296 config-0 atmospheres on B200 against 0.261 with three (74 registers);
// the items are chains of FP64 divisions, hidden by resident warps.
constexpr int DIFF_THREADS = 256;
constexpr int DIFF_LAYERS = 8;
__host__ __device__ inline size_t diff_block_smem_bytes(int ni) {
  constexpr int NR = DIFF_LAYERS + 2;
  return ((size_t)NR * (ni + 1) + ni + NR + 7 * NR + 3 * DIFF_LAYERS) * sizeof(double);
}

__global__ void __launch_bounds__(DIFF_THREADS, 4)
diffusion_rows_kernel(Batch B, const double* __restrict__ y, const double* __restrict__ atm, int flags,
                      const uint8_t* __restrict__ fix_mask, double* __restrict__ ws, double* __restrict__ resid,
                      int mode) {
  extern __shared__ __align__(16) double smem[];
  constexpr int LB = DIFF_LAYERS, NR = LB + 2;
  const int b = blockIdx.y, jb = blockIdx.x * LB;
  Geo g = geo_of(B, b);
  if (jb >= g.nz) return;
  const int ni = B.ni, nz = g.nz, rs = ni + 1;
  double* ys = smem;               // [NR][ni+1]: rows jb-1 .. jb+LB (0 outside [0, nz); padding 1.0)
  double* gas = ys + NR * rs;      // [ni]
  double* scal = gas + ni;         // [NR]: gas sums of those rows
  double* lay = scal + NR;         // [7][NR]: Kzz dzi vz Hpi Ti Tco g of those layers
  double* edd = lay + 7 * NR;      // [LB][3]: eddy A, B, C of the block's layers
  const AtmRef a = atm_ref(atm + g.atm, nz, ni);
  const WsView w = ws_view(ws, g, ni, B.ld);
  const double* yb = y + g.z0 * ni;
  const bool yk2 = mode == 2 && !resid;   // stage 2: rows of yk2 = y + k1/r
  const double r = ros2_r();
  for (int t = threadIdx.x; t < NR * rs; t += blockDim.x) {
    const int rr = t / rs, i = t % rs, jj = jb - 1 + rr;
    double v = 1.0;
    if (i < ni) {
      if (jj >= 0 && jj < nz) {
        v = yb[(int64_t)jj * ni + i];
        if (yk2) v = v + w.k1[(int64_t)jj * ni + i] / r;
      } else {
        v = 0.0;
      }
    }
    ys[t] = v;
  }
  for (int i = threadIdx.x; i < ni; i += blockDim.x) gas[i] = a.gas[i];
  for (int t = threadIdx.x; t < 7 * NR; t += blockDim.x) {
    const int f = t / NR, m = jb - 1 + t % NR;
    const double* src = f == 0 ? a.Kzz : f == 1 ? a.dzi : f == 2 ? a.vz : f == 3 ? a.Hpi : f == 4 ? a.Ti
                      : f == 5 ? a.Tco : a.g;
    lay[t] = (m >= 0 && m < nz) ? src[m] : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < NR) {
    const int jj = jb - 1 + (int)threadIdx.x;
    scal[threadIdx.x] = (jj >= 0 && jj < nz) ? pairwise_sum_masked(ys + threadIdx.x * rs, gas, ni) : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < LB) {
    const int l = threadIdx.x, j = jb + l;
    if (j < nz) {
      RowAcc E{};
      E.lay = lay;
      E.j0 = j - 1;
      E.base = jb - 1;
      E.S = NR;
      double A, Bc, C;
      eddy_row_t(E, nz, j, scal[l], scal[l + 1], scal[l + 2], A, Bc, C);
      edd[3 * l] = A;
      edd[3 * l + 1] = Bc;
      edd[3 * l + 2] = C;
    }
  }
  __syncthreads();
  const double use_vm = (flags & VB_USE_VM_MOL) ? 1.0 : 0.0;
  const double use_set = (flags & VB_USE_SETTLING) ? 1.0 : 0.0;
  for (int q = threadIdx.x; q < LB * ni; q += blockDim.x) {
    const int l = q / ni, i = q % ni, j = jb + l;
    if (j >= nz) continue;
    double Am, Bm, Cm;
    mol_row_t(row_acc(a, lay, ni, j, i, jb - 1, NR), nz, j, i, scal[l], scal[l + 1], scal[l + 2], use_vm,
                      use_set, Am, Bm, Cm);
    const double At = edd[3 * l] + Am;
    const double Bt = edd[3 * l + 1] + Bm;
    const double Ct = edd[3 * l + 2] + Cm;
    const double d = diffusion_term(a, nz, j, i, flags, At, Bt, Ct, ys[(l + 1) * rs + i], ys[l * rs + i],
                                    ys[(l + 2) * rs + i]);
    if (mode == 2) {
      (resid ? resid + g.z0 * ni : w.rmod)[(int64_t)j * ni + i] = d;
      continue;
    }
    if (mode == 0) w.rmod[(int64_t)j * ni + i] = d;
    w.aux[(int64_t)j * ni + i] = At;
    const bool fixed = mode == 0 && fix_mask && fix_mask[g.z0 * ni + (int64_t)j * ni + i];
    if (j < nz - 1) w.supn[(int64_t)j * ni + i] = mode == 1 ? Bt : (fixed ? 0.0 : -Bt);
    if (j > 0) w.subn[(int64_t)(j - 1) * ni + i] = mode == 1 ? Ct : (fixed ? 0.0 : -Ct);
  }
}

static cudaError_t launch_diffusion_rows(const Batch& B, const double* y, const double* atm, int flags,
                                         const uint8_t* fm, double* ws, double* resid, int mode, cudaStream_t st) {
  dim3 grid((B.nz + DIFF_LAYERS - 1) / DIFF_LAYERS, B.count);
  diffusion_rows_kernel<<<grid, DIFF_THREADS, diff_block_smem_bytes(B.ni), st>>>(B, y, atm, flags, fm, ws, resid,
                                                                                 mode);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- layer-vectorized stage 2
// The stage-2 right-hand side with one thread per layer instead of one CTA per
// layer: every term of a species list is then one coalesced load of a row of
// layers that the whole warp shares, in place of a dependent chain of table,
// shared-memory and L2 loads per lane. Two passes:
//  * lv_rates_kernel: the rate of every reaction slot at every layer of an
//    atmosphere at yk2 = y + k1/r (the state rows staged transposed in shared
//    memory; the rate constants k[r][z] read with the layers contiguous, the
//    reference's layout), into the rate region (rows [nr+1][nz_b]);
//  * lv_sums_kernel (a CTA per species and atmosphere, a thread per layer):
//    the species' loss and production sums, rmod = rhs(yk2) - 2/(r dt) k1.
// Each sum runs over the same terms, in the same order, with the same
// operations as in stage2_kernel, so the results are identical. (The same
// scheme for stage 1, with the rate derivatives staged too and the Jacobian
// rows summed per layer, measured slower than stage1_kernel on B200: 3.0 ms
// against 2.5 at 296 config-0 atmospheres; its scattered block-row stores
// and staging buffers cost more than the per-layer gathers.)
constexpr int LV_LAYERS = 128;         // layers of one thread group (a z-tile)
constexpr int LV_RATE_THREADS = 512;   // four groups; reactions dealt round the groups

__host__ __device__ inline size_t lv_rates_smem_bytes(int ni) {
  return (size_t)(ni + 1) * (LV_LAYERS + 1) * sizeof(double);
}

template <int TT>
__global__ void __launch_bounds__(LV_RATE_THREADS, 2)
lv_rates_kernel(NetDev net, Batch B, const double* __restrict__ y, const double* __restrict__ k,
                const double* __restrict__ atm, double* __restrict__ ws) {
  extern __shared__ __align__(16) double smem[];
  constexpr int RU = 4;   // rate constants loaded ahead
  const int b = blockIdx.y;
  const Geo g = geo_of(B, b);
  const int ni = B.ni, nzb = g.nz, R = B.nr + 1, S = LV_LAYERS + 1;
  const int r_lo = (int)((int64_t)R * blockIdx.x / gridDim.x);
  const int r_hi = (int)((int64_t)R * (blockIdx.x + 1) / gridDim.x);
  const double* yb = y + g.z0 * ni;
  const WsView w = ws_view(ws, g, ni, B.ld);
  const AtmRef a = atm_ref(atm + g.atm, nzb, ni);
  const double* kb = k + g.z0 * R;
  double* rate = B.rates + g.z0 * rates_region_doubles(B.nr);
  const double r = ros2_r();
  const int grp = threadIdx.x / LV_LAYERS, zl = threadIdx.x % LV_LAYERS, ngrp = blockDim.x / LV_LAYERS;
  double* yT = smem;   // [ni+1][S]: yk2 of species i at layer zl (row ni: the padding slot, 1.0)
  int any_lo = 0;      // the chunk's first slot in any_list (increasing)
  for (int n = net.n_any; n > 0;) {
    const int half = n / 2;
    const bool below = net.any_list[any_lo + half] < r_lo;
    any_lo += below ? half + 1 : 0;
    n = below ? n - half - 1 : half;
  }
  for (int zt = 0; zt < nzb; zt += LV_LAYERS) {
    const int nzt = min(LV_LAYERS, nzb - zt);
    __syncthreads();   // the previous tile's reads
    for (int e = threadIdx.x; e < nzt * ni; e += blockDim.x) {
      const int zz = e / ni, i = e - zz * ni;
      const int64_t q = (int64_t)(zt + zz) * ni + i;
      yT[i * S + zz] = yb[q] + w.k1[q] / r;   // stage2_kernel's expression
    }
    for (int zz = threadIdx.x; zz < LV_LAYERS; zz += blockDim.x) yT[ni * S + zz] = 1.0;
    __syncthreads();
    const int z = zt + zl;
    const bool on = zl < nzt;
    const double M = on ? a.M[z] : 0.0;
    for (int r0 = r_lo + grp; r0 < r_hi; r0 += RU * ngrp) {
      double kv[RU];
#pragma unroll
      for (int u = 0; u < RU; ++u) {
        const int rr = r0 + u * ngrp;
        kv[u] = (on && rr < r_hi) ? __ldcg(kb + (int64_t)rr * nzb + z) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < RU; ++u) {
        const int rr = r0 + u * ngrp;
        if (rr < r_hi) {
          const Slot sl = load_slot<TT>(net, rr);
          if (any_powers<TT>(sl)) continue;
          double yr[TT], d[TT];
#pragma unroll
          for (int s = 0; s < TT; ++s) yr[s] = yT[slot_species<TT>(sl, s) * S + zl];
          const double rt = rate_terms_p<TT, WholePowers>(yr, sl, kv[u], M, false, d);
          if (on) rate[(int64_t)rr * nzb + z] = rt;
        }
      }
    }
    // the slots that need pow, apart: the call's registers spilled in the loop
    // above (stage 2 of 64 atmospheres of 40 layers, 100 species and 3,300
    // reactions of four terms 0.529 ms so, 0.427 now)
    for (int q = any_lo + grp; q < net.n_any; q += ngrp) {
      const int rr = net.any_list[q];
      if (rr >= r_hi) break;
      const Slot sl = load_slot<TT>(net, rr);
      double yr[TT], d[TT];
#pragma unroll
      for (int s = 0; s < TT; ++s) yr[s] = yT[slot_species<TT>(sl, s) * S + zl];
      const double rt = rate_terms_any<TT>(yr, sl, on ? __ldcg(kb + (int64_t)rr * nzb + z) : 0.0, M, false, d);
      if (on) rate[(int64_t)rr * nzb + z] = rt;
    }
  }
}

__global__ void __launch_bounds__(LV_LAYERS)
lv_sums_kernel(NetDev net, Batch B, const double* __restrict__ dt, const uint8_t* __restrict__ fix_mask,
               double* __restrict__ ws) {
  __shared__ double coefs[MAX_COEF + 1];
  load_coefs(net, coefs);
  __syncthreads();
  const int i = blockIdx.x, b = blockIdx.y;
  const Geo g = geo_of(B, b);
  const int ni = B.ni, nzb = g.nz;
  const WsView w = ws_view(ws, g, ni, B.ld);
  const double* rate = B.rates + g.z0 * rates_region_doubles(B.nr);
  const double r = ros2_r();
  for (int zt = 0; zt < nzb; zt += LV_LAYERS) {
    const int z = zt + (int)threadIdx.x;
    if (z >= nzb) break;
    double part[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int e0 = net.sum_nptr[2 * i + t], e1 = net.sum_nptr[2 * i + t + 1];
      double acc = 0.0;
      if (net.coef_packed) {
#pragma unroll 8
        for (int e = e0; e < e1; ++e) {
          const uint32_t x = net.sum_nw[e];
          acc = acc + term_coef<true>(coefs, x) * rate[(int64_t)(x & 0xffffu) * nzb + z];
        }
      } else {
#pragma unroll 8
        for (int e = e0; e < e1; ++e) {
          const uint32_t x = net.sum_nw[e];
          acc = acc + term_coef<false>(coefs, x) * rate[(int64_t)(x & 0xffffu) * nzb + z];
        }
      }
      part[t] = acc;
    }
    // rmod holds the row's diffusion term (diffusion_rows_kernel)
    const int64_t q = (int64_t)z * ni + i;
    double v = (part[1] - part[0]) + w.rmod[q];
    if (fix_mask && fix_mask[g.z0 * ni + q]) v = 0.0;
    w.rmod[q] = v - (2.0 / (r * dt[b])) * w.k1[q];
  }
}

// ---------------------------------------------------------------- stage 2 by tiles of layers
// The stage-2 right-hand side of TZ consecutive layers of one atmosphere: the
// layers are the fastest lanes, so rate constants are read by sectors, a term
// is one word for eight lanes and eight neighbouring rates, and the rates
// never leave shared memory. The same terms in the same order as
// stage2_kernel's. The warps take quadruples of species lists (in the order of
// the groups, longest first) from a queue. Bound by the latency of the rate
// constants and of the longest lists at two CTAs per SM: 0.39 ms at 296
// atmospheres of 69 species and 120 layers, against 0.28 + 0.24 of the two
// thread-per-layer passes, which write and read every rate in global memory;
// 0.52 before the slots that need pow went ahead of the others.
constexpr int TZ = 8;
constexpr int TZ_THREADS = 512;

__host__ __device__ inline size_t tz_smem_bytes(int ni, int nr) {
  return (size_t)TZ * ((size_t)(nr + 1) + (ni + 1) + 2 * (size_t)ni) * sizeof(double);
}

template <bool PK>
__device__ __forceinline__ void tz_sums(const NetDev& net, const double* coef, const double* rate, int* queue,
                                        double* part) {
  const int lane = threadIdx.x & 31, z = lane % TZ;
  while (true) {
    int q = 0;
    if (lane == 0) q = atomicAdd(queue, 1);
    q = 4 * __shfl_sync(0xffffffffu, q, 0);
    if (q >= 2 * net.ni) break;
    q += lane / TZ;
    const uint32_t desc = net.gl_desc[q];
    const bool on = desc != ~0u;
    const int cnt = on ? (int)(desc & 0xffffu) : 0;
    const int len = __shfl_sync(0xffffffffu, cnt, 0);   // the first list is the longest
    const uint32_t* wp = net.gl_w + net.gl_base[q >> 5] + (q & 31);
    uint32_t w[GW];
    group_words(wp, len, w);
    double acc[1];
    gather_list<PK, 1>(coef, [&](int i) { return Vals<1>{{rate[i * TZ + z]}}; }, wp, len, cnt, w, acc);
    if (on) part[(desc >> 16) * TZ + z] = acc[0];
  }
}

template <int TT>
__global__ void __launch_bounds__(TZ_THREADS, 2)
stage2_tile_kernel(NetDev net, Batch B, const double* __restrict__ y, const double* __restrict__ k,
                   const double* __restrict__ dt, const double* __restrict__ atm,
                   const uint8_t* __restrict__ fix_mask, double* __restrict__ ws) {
  extern __shared__ __align__(16) double smem[];
  constexpr int RU = 4;   // rate constants loaded ahead
  const int b = blockIdx.y, j0 = TZ * blockIdx.x;
  const Geo g = geo_of(B, b);
  if (j0 >= g.nz) return;
  const int ni = B.ni, R = B.nr + 1, nl = min(TZ, g.nz - j0);
  double* rate = smem;            // [R][TZ]
  double* yT = rate + R * TZ;     // [ni+1][TZ]
  double* part = yT + (ni + 1) * TZ;   // [2 ni][TZ]
  const WsView w = ws_view(ws, g, ni, B.ld);
  const AtmRef a = atm_ref(atm + g.atm, g.nz, ni);
  const double* yb = y + (g.z0 + j0) * ni;
  const double* k1 = w.k1 + (int64_t)j0 * ni;
  const double r = ros2_r();
  __shared__ double coefs[MAX_COEF + 1];
  __shared__ int queue, slots;
  if (threadIdx.x == 0) queue = slots = 0;
  load_coefs(net, coefs);
  for (int e = threadIdx.x; e < nl * ni; e += blockDim.x) {
    const int z = e / ni, i = e - z * ni;
    yT[i * TZ + z] = yb[e] + k1[e] / r;   // stage2_kernel's expression
  }
  if (threadIdx.x < TZ) yT[ni * TZ + threadIdx.x] = 1.0;
  __syncthreads();
  // warps take blocks of RU quadruples of slots, after those that need pow (rates_t)
  const int lane = threadIdx.x & 31, z = lane % TZ, sub = lane / TZ, n_any = (net.n_any + 3) / 4;
  const bool on = z < nl;
  const double M = a.M[j0 + (on ? z : 0)];
  const double* kb = k + g.z0 * R + j0 + (on ? z : 0);
  while (true) {
    int q = 0;
    if (lane == 0) q = atomicAdd(&slots, 1);
    q = __shfl_sync(0xffffffffu, q, 0);
    const bool any = q < n_any;
    const int r0 = any ? 0 : 4 * RU * (q - n_any);
    if (r0 >= R) break;
    if (any) {
      if (4 * q + sub < net.n_any) {
        const int rr = net.any_list[4 * q + sub];
        const Slot S = load_slot<TT>(net, rr);
        double yr[TT], d[TT];
#pragma unroll
        for (int s = 0; s < TT; ++s) yr[s] = yT[slot_species<TT>(S, s) * TZ + z];
        rate[rr * TZ + z] = rate_terms_any<TT>(yr, S, __ldcg(kb + (int64_t)rr * g.nz), M, false, d);
      }
      __syncwarp();
      continue;
    }
    double kv[RU];
    Slot S[RU];
#pragma unroll
    for (int u = 0; u < RU; ++u) {
      const int rr = min(r0 + 4 * u + sub, R - 1);
      kv[u] = __ldcg(kb + (int64_t)rr * g.nz);
      if (TT <= RX_TERMS) S[u] = load_slot<TT>(net, rr);
    }
#pragma unroll
    for (int u = 0; u < RU; ++u) {
      const int rr = r0 + 4 * u + sub;
      if (TT > RX_TERMS) S[u] = load_slot<TT>(net, min(rr, R - 1));
      if (rr < R && !any_powers<TT>(S[u])) {
        double yr[TT], d[TT];
#pragma unroll
        for (int s = 0; s < TT; ++s) yr[s] = yT[slot_species<TT>(S[u], s) * TZ + z];
        rate[rr * TZ + z] = rate_terms_p<TT, WholePowers>(yr, S[u], kv[u], M, false, d);
      }
    }
  }
  __syncthreads();
  if (net.coef_packed)
    tz_sums<true>(net, coefs, rate, &queue, part);
  else
    tz_sums<false>(net, coefs, rate, &queue, part);
  __syncthreads();
  const uint8_t* fm = fix_mask ? fix_mask + (g.z0 + j0) * ni : nullptr;
  double* rmod = w.rmod + (int64_t)j0 * ni;   // holds the rows' diffusion terms (diffusion_rows_kernel)
  const double c = 2.0 / (r * dt[b]);
  for (int e = threadIdx.x; e < nl * ni; e += blockDim.x) {
    const int zz = e / ni, i = e - zz * ni;
    double v = (part[(2 * i + 1) * TZ + zz] - part[2 * i * TZ + zz]) + rmod[e];
    if (fm && fm[e]) v = 0.0;
    rmod[e] = v - c * k1[e];
  }
}

static cudaError_t launch_stage2_tiles(const NetDev& net, const Batch& B, const double* y, const double* k,
                                       const double* dt, const double* atm, const uint8_t* fm, double* ws,
                                       cudaStream_t st) {
  const size_t sm = tz_smem_bytes(B.ni, B.nr);
  dim3 grid((B.nz + TZ - 1) / TZ, B.count);
  cudaError_t e = cudaSuccess;
  auto go = [&](auto kern) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e == cudaSuccess) kern<<<grid, TZ_THREADS, sm, st>>>(net, B, y, k, dt, atm, fm, ws);
  };
  switch (net.T) {
    case 1: go(stage2_tile_kernel<1>); break;
    case 2: go(stage2_tile_kernel<2>); break;
    case 3: go(stage2_tile_kernel<3>); break;
    case 4: go(stage2_tile_kernel<4>); break;
    case 5: go(stage2_tile_kernel<5>); break;
    case 6: go(stage2_tile_kernel<6>); break;
    case 7: go(stage2_tile_kernel<7>); break;
    default: go(stage2_tile_kernel<8>); break;
  }
  return cudaGetLastError();
}

static int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    sms = 148;
  return sms;
}

// Reaction chunks per atmosphere of lv_rates_kernel: about two waves of
// three 512-thread CTAs per SM, at least 8 reaction slots per chunk.
static int lv_rate_chunks(const Batch& B) {
  const int want = (6 * sm_count() + B.count - 1) / B.count;
  return std::max(1, std::min(want, (B.nr + 1) / 8));
}

static cudaError_t launch_lv_stage2(const NetDev& net, const Batch& B, const double* y, const double* k,
                                    const double* dt, const double* atm, const uint8_t* fm, double* ws,
                                    cudaStream_t st) {
  const size_t sm = lv_rates_smem_bytes(B.ni);
  dim3 grid(lv_rate_chunks(B), B.count);
  cudaError_t e = cudaSuccess;
  auto go = [&](auto kern) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e == cudaSuccess) kern<<<grid, LV_RATE_THREADS, sm, st>>>(net, B, y, k, atm, ws);
  };
  switch (net.T) {
    case 1: go(lv_rates_kernel<1>); break;
    case 2: go(lv_rates_kernel<2>); break;
    case 3: go(lv_rates_kernel<3>); break;
    case 4: go(lv_rates_kernel<4>); break;
    case 5: go(lv_rates_kernel<5>); break;
    case 6: go(lv_rates_kernel<6>); break;
    case 7: go(lv_rates_kernel<7>); break;
    default: go(lv_rates_kernel<8>); break;
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  lv_sums_kernel<<<dim3(B.ni, B.count), LV_LAYERS, 0, st>>>(net, B, dt, fm, ws);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- launchers
// Layers per CTA of the stage-1 assembly (VbTuning.stage1_layers, or by size).
// Two layers read every gather word, descriptor and rate-constant sector once
// for both, but halve the CTAs that hide each other's phases. Measured on
// B200, one / two layers, stage 1 with the diffusion rows: networks whose
// one-layer CTAs (a layer's drates) no longer fit four to an SM: 1.91 / 1.73 ms
// (89 species, 2,000 reactions, 19,200 layers), 0.232 / 0.197 (128, 3,000,
// 960 layers); that fit four but leave L1 under 40 KB: 2.02 / 1.98 (69, 1,400,
// 35,520 layers) yet 0.149 / 0.152 at 1,920 layers; smaller ones 0.266 / 0.269
// (64, 1,000) and 0.251 / 0.278 (30, 370, 256 atmospheres of 43 layers).
static int stage1_layers(const NetDev& net, const Batch& B) {
  if (B.stage1_layers) return B.stage1_layers;
  const size_t per_sm = 228 * 1024, l1 = 40 * 1024;
  const size_t cta = stage1_smem_bytes(B.ni, B.nr, net.T, 1) + (MAX_COEF + 1) * sizeof(double) + 1024;
  if (stage1_smem_bytes(B.ni, B.nr, net.T, 2) > per_sm - 4096 || 4 * cta + l1 <= per_sm) return 1;
  const int64_t least = 4 * cta > per_sm ? 4 : 16;   // layers per SM
  return (int64_t)B.count * B.nz >= least * sm_count() ? 2 : 1;
}

template <int NL>
static cudaError_t launch_stage1_t(const NetDev& net, const Batch& B, const double* y, const double* k,
                                   const double* dt, const double* atm, int flags, const uint8_t* fm, double* ws,
                                   cudaStream_t st, const double* adj_v) {
  const size_t sm = stage1_smem_bytes(B.ni, B.nr, net.T, NL);
  cudaError_t e = cudaFuncSetAttribute(stage1_kernel<NL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return cudaGetLastError();   // too large a layer; leaves no error behind
  stage1_kernel<NL><<<dim3((B.nz + NL - 1) / NL, B.count), NL * LAYER_THREADS, sm, st>>>(net, B, y, k, dt, atm, flags,
                                                                                         fm, ws, adj_v);
  return cudaGetLastError();
}

cudaError_t launch_stage1(const NetDev& net, const Batch& B, const double* y, const double* k,
                          const double* dt, const double* atm, int flags, const uint8_t* fm, double* ws,
                          cudaStream_t st, const double* adj_v) {
  cudaError_t e = launch_diffusion_rows(B, y, atm, flags, fm, ws, nullptr, adj_v ? 1 : 0, st);
  if (e != cudaSuccess) return e;
  return stage1_layers(net, B) == 2 ? launch_stage1_t<2>(net, B, y, k, dt, atm, flags, fm, ws, st, adj_v)
                                    : launch_stage1_t<1>(net, B, y, k, dt, atm, flags, fm, ws, st, adj_v);
}

template <int NL>
static cudaError_t launch_stage2_t(const NetDev& net, const Batch& B, const double* y, const double* k,
                                   const double* dt, const double* atm, const uint8_t* fm, double* ws,
                                   cudaStream_t st, double* resid) {
  const size_t sm = stage2_smem_bytes(B.ni, B.nr, NL);
  cudaError_t e = cudaFuncSetAttribute(stage2_kernel<NL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return cudaGetLastError();
  stage2_kernel<NL><<<dim3((B.nz + NL - 1) / NL, B.count), NL * LAYER_THREADS, sm, st>>>(net, B, y, k, dt, atm, fm, ws,
                                                                                         resid);
  return cudaGetLastError();
}

// Tiles where their rates fit shared memory and two CTAs per SM have work;
// fewer layers leave SMs idle that the reaction chunks of the thread-per-layer
// passes fill. Measured on B200, thread per layer / tiles, stage 2 with the
// diffusion rows: 0.63 / 0.51 ms (296 atmospheres of 69 species, 120 layers),
// 0.72 / 0.51 (128 of 89, 150 layers), 0.083 / 0.041 (33 of 45, 97 layers).
bool stage2_tiles(const Batch& B) {
  return tz_smem_bytes(B.ni, B.nr) <= 220 * 1024 && (int64_t)B.count * ((B.nz + TZ - 1) / TZ) >= 2 * sm_count();
}

cudaError_t launch_stage2(const NetDev& net, const Batch& B, const double* y, const double* k,
                          const double* dt, const double* atm, int flags, const uint8_t* fm, double* ws,
                          cudaStream_t st, double* resid) {
  cudaError_t e = launch_diffusion_rows(B, y, atm, flags, fm, ws, resid, 2, st);
  if (e != cudaSuccess) return e;
  if (!resid && stage2_tiles(B)) return launch_stage2_tiles(net, B, y, k, dt, atm, fm, ws, st);
  if (!resid && B.stage1_layers == 2) return launch_stage2_t<2>(net, B, y, k, dt, atm, fm, ws, st, resid);
  if (!resid && B.rates) return launch_lv_stage2(net, B, y, k, dt, atm, fm, ws, st);
  return launch_stage2_t<1>(net, B, y, k, dt, atm, fm, ws, st, resid);
}

cudaError_t launch_chem(const NetDev& net, int batch, int nz, const double* y, const double* M,
                        const double* k, double* dydt, double* jac, cudaStream_t st) {
  size_t sm = chem_smem_bytes(net.ni, net.nr, net.T, jac != nullptr);
  auto kern = jac ? chem_kernel<true> : chem_kernel<false>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  dim3 grid(nz, batch);
  kern<<<grid, LAYER_THREADS, sm, st>>>(net, nz, y, M, k, dydt, jac);
  return cudaGetLastError();
}

cudaError_t launch_diffusion(int batch, int nz, int ni, const double* y, const double* atm, int flags,
                             double* diff, double* diag_d, double* sup_d, double* sub_d,
                             cudaStream_t st) {
  size_t sm = layer_smem_bytes(ni);
  dim3 grid(nz, batch);
  diffusion_kernel<<<grid, LAYER_THREADS, sm, st>>>(nz, ni, y, atm, flags, diff, diag_d, sup_d, sub_d);
  return cudaGetLastError();
}

}  // namespace vb
