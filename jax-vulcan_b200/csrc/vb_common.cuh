// Shared device-side definitions of the B200 Ros2 kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "vulcan_b200.h"

namespace vb {

constexpr int GL_SHORT = 4;   // longest Jacobian list with code of its own (reason: vb_chem.cu, gather_short)
constexpr int RX_TERMS = 6;   // reactant slots that fit a packed reaction word

// Code of a stoichiometry: 0, 1, 2, or 3 for any other value.
__host__ __device__ __forceinline__ uint32_t st_code(double st) {
  return st == 0.0 ? 0u : st == 1.0 ? 1u : st == 2.0 ? 2u : 3u;
}


// Device-resident network tables (reference chem.py:28-80 plus gather tables).
struct NetDev {
  int ni, nr, T;                 // species, reaction slots (rows nr+1), max_terms
  const int32_t* r_idx;          // [nr+1][T]
  const int32_t* p_idx;          // [nr+1][T]
  const double* r_st;            // [nr+1][T]
  const double* p_st;            // [nr+1][T]
  const uint8_t* three;          // [nr+1]
  // Reaction slot in one word (T <= RX_TERMS): reactant index s in byte s, its
  // stoichiometry's code (st_code) at bits 48 + 2 s, the three-body flag at bit 60.
  const uint64_t* rx;            // [nr+1]
  // Reactions with a stoichiometry of code 3 (their powers take pow).
  const int32_t* any_list;       // [n_any]
  int n_any;
  // Gather tables, one 32-bit word per term: the low 16 bits index a rate
  // (species lists: reaction r) or a drate slot (Jacobian: r*T+s), the high 16
  // bits give the coefficient: the top half of the double's high word where
  // every coefficient of the network is zero below it (coef_packed; whole and
  // half stoichiometries are), else its id in coef_tab (<= 256 distinct ones).
  // The lists, in groups of 32, by falling term count (ties: increasing index):
  // * the 2 ni species lists, t = 2 i (loss) or 2 i + 1 (production) of
  //   species i: the (r*T+s) slots whose reactant (loss) or product index is
  //   i, in increasing flat order (segment_sum order), with r_st or p_st;
  // * the ni*ni Jacobian entries: the contributions (r, o, s) in increasing
  //   flat order (r*2T + o)*T + s (chem.py:193-207 scatter order), with
  //   -r_st[r][o] (o < T) or p_st[r][o-T].
  // Groups [0, gl_sums) hold the species lists, [gl_sums, gl_diag) the
  // diagonal entries, [gl_diag, gl_long) the off-diagonal entries of more than
  // GL_SHORT terms, [gl_long, gl_groups) the others, by increasing entry and
  // each filled up to GL_SHORT terms with the index (nr+1)*T (a drate of 0) and
  // a finite coefficient, which change no sum. The last group of a kind has
  // lanes whose descriptor is ~0. The words of a group are interleaved and
  // padded (with 0) to its longest list: term k of lane l of group g at
  // gl_w[gl_base[g] + 32 k + l], so a warp that holds a group loads one line
  // per term.
  const uint32_t* gl_base;       // [gl_groups + 1]
  const uint32_t* gl_desc;       // [32 gl_groups]: count | t << 16, or count | row << 16 | col << 23
  const uint32_t* gl_w;
  int gl_sums, gl_diag, gl_long, gl_groups;
  const double* coef_tab;        // [n_coef]
  int n_coef, coef_packed;
  // The species lists in natural order, for the layer-vectorized stage 2
  // (one thread per layer, every term of a list read by the whole warp):
  // list t (2 i loss, 2 i + 1 production) at sum_nw[sum_nptr[t] .. sum_nptr[t+1]).
  const int32_t* sum_nptr;       // [2 ni + 1]
  const uint32_t* sum_nw;
};

constexpr int LAYER_THREADS = 256;
constexpr int MAX_COEF = 256;   // distinct stoichiometric coefficients of a network (and 0.0 for filled-up lists)

// Term word of a gather table: index (low 16 bits) and the coefficient's
// high half-word or id.
__host__ __device__ __forceinline__ uint32_t term_word(int idx, int code) {
  return (uint32_t)idx | ((uint32_t)code << 16);
}

// Offsets (in doubles) of the fields of one atmosphere in the atm blob.
struct AtmOff {
  int64_t Kzz, dzi, vz, Hpi, Ti, Tco, g, M, Dzz, vm, vs, ms, alpha, top, bot, vdep, gas;
};

__host__ __device__ inline AtmOff atm_offsets(int nz, int ni) {
  AtmOff o;
  int64_t NZ = nz, NI = ni;
  o.Kzz = 0; o.dzi = NZ; o.vz = 2 * NZ; o.Hpi = 3 * NZ; o.Ti = 4 * NZ; o.Tco = 5 * NZ;
  o.g = 6 * NZ; o.M = 7 * NZ;
  o.Dzz = 8 * NZ; o.vm = o.Dzz + NZ * NI; o.vs = o.vm + NZ * NI;
  o.ms = o.vs + NZ * NI; o.alpha = o.ms + NI; o.top = o.alpha + NI; o.bot = o.top + NI;
  o.vdep = o.bot + NI; o.gas = o.vdep + NI;
  return o;
}

// Per-atmosphere geometry of a (possibly ragged) batch.
struct Batch {
  int count;          // atmospheres
  int nz;             // layers (uniform) or maximum layers (ragged)
  int ni;
  int nr;             // reaction slots (k has nr+1 rows)
  int ld;             // row stride of stored inverse blocks (ni rounded up to even)
  const int64_t* zoff;  // [count+1] prefix sums of layers, or nullptr (uniform)
  // launch shapes chosen by the network's tuning (VbTuning; 0 = automatic)
  int factor_kernel = 0;   // 1 blocked tensor-core, 2 by panels, 3 pipelined, 4 paired
  int factor_ctas = 0;     // CTAs per SM of the factor (1 or 2, where both fit)
  int sweep_stages = 0;    // bulk-copy ring depth of the sweeps (1..3; 0: as deep as fits)
  int stage1_layers = 0;   // layers per stage-1 CTA (1 or 2)
  // rate region of the layer-vectorized stage 2 (rates_region_doubles per
  // layer), or nullptr: the per-layer stage-2 kernel
  double* rates = nullptr;
};

// Doubles per layer of the rate region: the rate of every reaction slot, rows
// [nr+1][nz_b] per atmosphere (layers contiguous).
__host__ __device__ inline int64_t rates_region_doubles(int nr) { return (int64_t)nr + 1; }

struct Geo {
  int nz;
  int64_t z0;        // first layer of this atmosphere in the packed layer axis
  int64_t atm;       // blob offset (doubles)
  int64_t ws;        // workspace offset (doubles)
};

// Workspace doubles per layer: inverse block + rmod + k1 + sup_neg + sub_neg +
// spare, rounded up to 16 doubles so every atmosphere's blocks start on a
// 128-byte boundary (bulk copies need 16-byte aligned addresses and sizes).
__host__ __device__ inline int64_t ws_per_layer(int ni, int ld) {
  return (((int64_t)ni * ld + 5 * (int64_t)ni) + 15) & ~(int64_t)15;
}

__device__ __forceinline__ Geo geo_of(const Batch& B, int b) {
  Geo g;
  if (B.zoff) {
    g.z0 = B.zoff[b];
    g.nz = (int)(B.zoff[b + 1] - g.z0);
  } else {
    g.z0 = (int64_t)b * B.nz;
    g.nz = B.nz;
  }
  g.atm = g.z0 * (8 + 3 * (int64_t)B.ni) + (int64_t)b * 6 * B.ni;
  g.ws = g.z0 * ws_per_layer(B.ni, B.ld);
  return g;
}

// Workspace sub-arrays of one atmosphere (all doubles).
struct WsView {
  double* inv;   // [nz][ni][ld]
  double* rmod;  // [nz][ni]  forward-eliminated right-hand side
  double* k1;    // [nz][ni]
  double* supn;  // [nz][ni]  (first nz-1 rows used): negated super-diagonal (solver's sup_d)
  double* subn;  // [nz][ni]  negated sub-diagonal (solver's sub_d)
  double* aux;   // [nz][ni]
};

__device__ __forceinline__ WsView ws_view(double* ws, const Geo& g, int ni, int ld) {
  WsView v;
  v.inv = ws + g.ws;
  int64_t blk = (int64_t)g.nz * ni * ld;
  int64_t vec = (int64_t)g.nz * ni;
  v.rmod = v.inv + blk;
  v.k1 = v.rmod + vec;
  v.supn = v.k1 + vec;
  v.subn = v.supn + vec;
  v.aux = v.subn + vec;
  return v;
}

__host__ __device__ inline int round_even(int n) { return (n + 1) & ~1; }

// ---- mixed-precision region of the Ros2 step (after the FP64 workspace):
// per atmosphere, [nz][ni][ldf] FP32 inverses of the row-equilibrated
// eliminated blocks (ldf = ni rounded up to 4, so each block is a multiple of
// 16 bytes), then [nz][ni] row scales r (A'^{-1} = X diag(r)), then [nz][ni]
// scratch (the forward-eliminated residual of a refinement pass).
__host__ __device__ inline int round4(int n) { return (n + 3) & ~3; }
__host__ __device__ inline int64_t mx_bytes_per_layer(int ni) {
  return (int64_t)ni * round4(ni) * 4 + 16 * (int64_t)ni;
}
struct MxView {
  float* X;      // [nz][ni][ldf]
  double* rs;    // [nz][ni]
  double* tmp;   // [nz][ni]
};
__host__ __device__ inline MxView mx_view(void* mx, int64_t z0, int nz, int ni) {
  char* base = static_cast<char*>(mx) + z0 * mx_bytes_per_layer(ni);
  MxView v;
  v.X = reinterpret_cast<float*>(base);
  v.rs = reinterpret_cast<double*>(base + (int64_t)nz * ni * round4(ni) * 4);
  v.tmp = v.rs + (int64_t)nz * ni;
  return v;
}

// ---------------------------------------------------------------- bulk copies
// Global -> shared bulk copies (cp.async.bulk, no multicast) completed on an
// mbarrier. Every wait is bounded: a wait that gives up reports false and the
// caller sets VB_STATUS_WATCHDOG.
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// 8-byte asynchronous copy global -> shared (both 8-byte aligned).
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long limit) {
  for (long long it = 0; it < limit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
constexpr long long WAIT_LIMIT = 1ll << 22;

// mbarriers as intra-CTA producer/consumer signals (no async copies): an
// arrival (release) per producing thread, a bounded wait (acquire) that also
// gives up as soon as another warp has raised *abort.
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_inval(uint64_t* bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_wait_or_abort(uint64_t* bar, uint32_t parity, long long limit,
                                                   const volatile int* abort) {
  for (long long it = 0; it < limit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (*abort) return false;
  }
  return false;
}

// a / b. A zero numerator (no wind, no settling, no molecular diffusion; opaque
// layers without beam or flux) over a finite nonzero b takes the product, whose
// value and sign are the quotient's, instead of the division's out-of-range
// path: at 296 atmospheres of 69 species and 120 layers without molecular
// diffusion the diffusion rows took 0.239 ms with that path and 0.117 without.
__device__ __forceinline__ double quot(double a, double b) {
  return a == 0.0 && b != 0.0 && fabs(b) <= 1.7976931348623157e308 ? a * b : a / b;
}

// Ros2 constants (reference jax_step.py:257-258).
__device__ __forceinline__ double ros2_r() { return 1.0 + 1.0 / sqrt(2.0); }

}  // namespace vb
