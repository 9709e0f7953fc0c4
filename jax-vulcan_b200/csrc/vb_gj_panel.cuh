// Block inverses of the block-Thomas factor by panel Gauss-Jordan elimination,
// one CTA per atmosphere (device code shared by the kernels of vb_thomas.cu).
#pragma once
#include <cuda_runtime.h>

#include "vb_common.cuh"

namespace vb {

// Pivot choice of every factor kernel. The key of a candidate row is the top
// 24 bits of |v| (exponent and the leading 13 mantissa bits in FP64, 16 in
// FP32) above 255 - row, so one 32-bit max reduction over the warp names the
// pivot row: the largest magnitude to within a relative 2^-13 (FP64) or 2^-16
// (FP32), the lowest row among those (threshold partial pivoting with threshold
// 1 - 2^-13; strict partial pivoting takes the exact maximum, at the price of a
// second reduction, ballots and shuffles on the pivot chain). The magnitude
// bits are shifted out of the sign and raised so that infinity, the largest,
// takes the top value; NaN wraps around below zero's and is brought to it (a
// NaN counts as magnitude 0). Two integer instructions: testing for NaN with a
// double comparison per row cost 160 of a step's 475 cycles. Rows that may not
// pivot (pivoted, padding) take key 0, below every candidate (row <= 127, so a
// candidate's low byte is >= 128).
__device__ __forceinline__ unsigned pivot_mag(double v) {
  return max(((unsigned)__double2hiint(v) << 1) + 0x001fff00u, 0x001fff00u);
}
__device__ __forceinline__ unsigned pivot_mag(float v) {
  return max((__float_as_uint(v) << 1) + 0x00ffff00u, 0x00ffff00u);
}
template <typename R>
__device__ __forceinline__ unsigned pivot_key32(R v, int row) {
  return (pivot_mag(v) & 0xffffff00u) | (unsigned)(255 - row);
}
// Largest key of a lane's rows (two at a time: one instruction).
template <int N>
__device__ __forceinline__ unsigned key_max(const unsigned (&k)[N]) {
  unsigned m = k[0];
#pragma unroll
  for (int r = 1; r + 1 < N; r += 2) m = __vimax3_u32(m, k[r], k[r + 1]);
  return N % 2 == 0 ? max(m, k[N - 1]) : m;
}
__device__ __forceinline__ int pivot_row(unsigned kmax) { return 255 - (int)(kmax & 255u); }

// Zero with the sign of v.
__device__ __forceinline__ double zero_as(double v) {
  return __hiloint2double(__double2hiint(v) & (int)0x80000000u, 0);
}
__device__ __forceinline__ float zero_as(float v) { return __uint_as_float(__float_as_uint(v) & 0x80000000u); }

// Correctly rounded reciprocal (the value of 1 / x).
__device__ __forceinline__ double rcp_rn(double x) { return __drcp_rn(x); }
__device__ __forceinline__ float rcp_rn(float x) { return __frcp_rn(x); }

// Power of two s with s * m in [1, 2) for a finite m > 0 (1 otherwise).
__device__ __forceinline__ double pow2_scale(double m) {
  if (!(m > 0.0) || !isfinite(m)) return 1.0;
  int e;
  frexp(m, &e);               // m = f 2^e, f in [0.5, 1)
  return ldexp(1.0, 1 - e);   // s m = 2 f in [1, 2)
}

// Two values of the factor's element type handed over in one shared-memory access.
template <typename R> struct Pair;
template <> struct Pair<double> { using T = double2; };
template <> struct Pair<float> { using T = float2; };

// Pair store to shared memory where `on` holds (a predicated instruction, not
// a branch: the arithmetic around it stays in one basic block).
__device__ __forceinline__ void st_pair_if(uint32_t addr, double x, double y, bool on) {
  asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %3, 0;\n @q st.shared.v2.f64 [%0], {%1, %2};\n}" ::"r"(addr),
               "d"(x), "d"(y), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void st_pair_if(uint32_t addr, float x, float y, bool on) {
  asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %3, 0;\n @q st.shared.v2.f32 [%0], {%1, %2};\n}" ::"r"(addr),
               "f"(x), "f"(y), "r"((int)on)
               : "memory");
}

// Shared-memory plan of panel_factor_atmosphere (carved in this order, each
// piece on a 16-byte boundary).
template <int RPL, int CPW, int NW, typename R>
struct PGJ {
  static constexpr int NPR = 32 * RPL;          // row capacity (lane l holds rows l + 32 r)
  static constexpr int NPC = CPW * NW;          // column capacity (warp w holds columns w*CPW + c)
  static constexpr int CPWP = (CPW + 1) & ~1;   // stride of a stored pivot row (pairs)
  static constexpr size_t MS = (size_t)CPW * NPR;    // multipliers of a panel
  static constexpr size_t US = 2 * (size_t)CPWP;     // a warp's pivot-row hand-over (2 parities)
  __host__ __device__ static size_t al(size_t x) { return (x + 15) & ~(size_t)15; }
  static size_t smem_bytes(int n, int ld, bool dpf, int li = 0) {
    const size_t blk = (size_t)n * ld, iblk = (size_t)n * (li ? li : ld);
    return al(iblk * sizeof(R))                       // Ib: the inverse of the layer (natural order, stride li)
           + (dpf ? al(blk * sizeof(double)) : 0)     // Db: the next diagonal block, prefetched
           + al(2 * NPC * sizeof(double))             // rsc: row scales of this and the previous layer (EQ)
           + al(NPR * sizeof(R))                      // rps: 1 / pivot of each row
           + al(6 * NPR * sizeof(double))             // cpl: sup_d[j], sub_d[j], rhs[j+1] (2 parities of j)
           + al(2 * NPR * sizeof(double))             // vecs: right-hand side ping-pong
           + al(NPC * sizeof(int))                    // pivs: pivot row of each step
           + al(NPR * sizeof(int))                    // qs: step of each pivot row (-1: not pivoted yet)
           + 16                                       // mbarrier of the prefetch
           + al(2 * MS * sizeof(R))                   // Mb: multipliers of a panel's steps (2 parities)
           + al(NW * US * sizeof(R));                 // Ub: pivot-row hand-over, a slot per warp and parity
  }
};

// Factor all layers of one atmosphere by Gauss-Jordan inversion of each
// Schur-updated diagonal block. On entry Din[j] holds D_j (row stride ld); on
// exit out[j] holds A'_j^{-1}; with rhs != nullptr the first sweep of the
// right-hand side rhs[nz][ni] is done in place (solver.py:73-88).
//
// The reference inverts each block by lu_factor then lu_solve(LU, I)
// (solver.py:46-48). Here the inverse comes from one serial chain of ni
// Gauss-Jordan steps instead of three (factor, forward and back
// substitution). Gauss-Jordan bounds the left residual |X B - I| of the
// inverse X of the matrix B it eliminates on. With tr set the elimination
// runs on the transposed block B = A'^T (partial pivoting within a row of
// A'), so X = A'^{-1} has a small right residual |A' X - I| as the
// reference's lu_solve(LU, I) columns do: what solves x = X b need (the Ros2
// step; on the stiff config-0 draw eliminating on A' itself left the block
// solve's normwise backward error at 4e-12 instead of 7e-15). Without tr it
// runs on B = A' (partial pivoting within a column, as lu_factor), for
// callers that solve with X^T (the transposed sweeps of the adjoint), which
// need |X A' - I| small.
//  * Tile in registers: lane l holds rows l + 32 r (r < RPL), warp w columns
//    w*CPW + c (c < CPW) of B. No row exchanges: row p_k is the pivot row
//    of step k. Pivot rows are not normalised during the elimination (row i
//    carries the factor piv_i of its own step), so every element update is
//    one FMA
//        S[i][:] -= m_i S[p][:],   m_i = S[i][k] / piv_k  (m_p = 0),
//    column k becomes -m_i (row p: 1), and each row is scaled by 1/piv_i at
//    the end. The stored result T satisfies B^{-1}[q(i)][p_m] = T[i][m]
//    (q(i): the step whose pivot row is i), applied (transposed back when
//    tr) by the scatter into Ib.
//  * EQ (transposed orientation): every row of A'_j is scaled by a power of
//    two bringing its largest magnitude to [1, 2) before the elimination
//    (row equilibration, exact); the stored inverse is X = (R A'_j)^{-1},
//    the scales go to rs_out, and A'_j^{-1} = X diag(r).
//  * li: row stride of Ib and of the stored inverses (ld when 0).
template <int RPL, int CPW, int NW, bool DPF, typename R, bool EQ>
__device__ __forceinline__ void panel_factor_atmosphere(int nz, int n, int ld, const double* Din, R* out,
                                                        const double* __restrict__ supn,
                                                        const double* __restrict__ subn, double* rhs, bool tr,
                                                        int32_t* status, char* smem_raw, long long wlim, int li,
                                                        double* rs_out) {
  using G = PGJ<RPL, CPW, NW, R>;
  using R2 = typename Pair<R>::T;
  constexpr int NPR = G::NPR, CPWP = G::CPWP, NPC = G::NPC;
  static_assert(CPW >= 2 && NW >= 2, "a panel's hand-over uses two slots; one warp eliminates while others finish");
  if (li == 0) li = ld;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned FULL = 0xffffffffu;
  const int blk = n * ld, iblk = n * li;
  char* sp = smem_raw;
  auto take = [&](size_t bytes) {
    char* q = sp;
    sp += G::al(bytes);
    return q;
  };
  R* Ib = reinterpret_cast<R*>(take((size_t)iblk * sizeof(R)));
  double* Db = DPF ? reinterpret_cast<double*>(take((size_t)blk * sizeof(double))) : nullptr;
  double* rsc = reinterpret_cast<double*>(take(2 * NPC * sizeof(double)));
  R* rps = reinterpret_cast<R*>(take(NPR * sizeof(R)));
  double* cpl = reinterpret_cast<double*>(take(6 * NPR * sizeof(double)));
  double* vecs = reinterpret_cast<double*>(take(2 * NPR * sizeof(double)));
  int* pivs = reinterpret_cast<int*>(take(NPC * sizeof(int)));
  int* qs = reinterpret_cast<int*>(take(NPR * sizeof(int)));
  uint64_t* bar = reinterpret_cast<uint64_t*>(take(16));
  R* Mb = reinterpret_cast<R*>(take(2 * G::MS * sizeof(R)));
  R* Ub = reinterpret_cast<R*>(take(NW * G::US * sizeof(R)));
  const uint32_t dbytes = (uint32_t)(blk * sizeof(double));
  int st_local = 0;

  for (int e = threadIdx.x; e < iblk; e += NW * 32) Ib[e] = R(0);   // the padding columns stay 0
  if (rhs)
    for (int i = threadIdx.x; i < n; i += NW * 32) vecs[i] = rhs[i];
  if (DPF && threadIdx.x == 0) mbar_init(bar, 1);
  __syncthreads();
  if (DPF && threadIdx.x == 0) {
    mbar_expect_tx(bar, dbytes);
    bulk_g2s(Db, Din, dbytes, bar);
  }

  R a[RPL][CPW];

  // The pivot steps of panel q (columns q CPW + s), run by the warp that owns
  // them from its registers with warp-level communication only: argmax by
  // redux.sync, pivot value by a shuffle, pivot row through the warp's
  // hand-over slot (two by step parity: one __syncwarp per step). The columns
  // rotate through the registers: the step's column is always slot 0 and every
  // update writes one slot lower, so the step loop is not unrolled by column.
  // The multipliers go to Mb (parity of q) for the other warps.
  auto factor_panel = [&](int q) {
    const int k0 = q * CPW, cnt = min(CPW, n - k0);
    R* Mq = Mb + (q & 1) * G::MS;
    R* hs = Ub + warp * G::US;
    // key of row r: the shifted magnitude under msk above cc (pivot_key_of);
    // both are 0 for the rows that may not pivot: pivoted before, or padding
    unsigned msk[RPL], cc[RPL];
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int i = lane + 32 * r;
      const bool free_row = i < n && qs[i] < 0;
      msk[r] = free_row ? 0xffffff00u : 0u;
      cc[r] = free_row ? 255u - (unsigned)i : 0u;
    }
    // Software pipeline: t is the step's column, up to date; the columns after
    // it still wait for the previous step (multipliers m, pivot row prow),
    // applied while the argmax is in flight; w is the column the previous step
    // finished.
    R t[RPL], w[RPL], m[RPL], prow[CPWP];
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      t[r] = a[r][0];
      w[r] = a[r][CPW - 1];
      m[r] = R(0);
    }
#pragma unroll
    for (int c2 = 0; c2 < CPWP; ++c2) prow[c2] = R(0);
#pragma unroll 1
    for (int s = 0; s < cnt; ++s) {
      unsigned kr[RPL];
#pragma unroll
      for (int r = 0; r < RPL; ++r) kr[r] = (pivot_mag(t[r]) & msk[r]) | cc[r];
      const unsigned km = key_max(kr);
      const unsigned kx = __reduce_max_sync(FULL, km);
      R vb = t[0];   // this lane's candidate
#pragma unroll
      for (int r = 1; r < RPL; ++r) vb = kr[r] == km ? t[r] : vb;
#pragma unroll
      for (int c2 = 1; c2 < CPW - 1; ++c2)
#pragma unroll
        for (int r = 0; r < RPL; ++r) a[r][c2 - 1] = fma(-m[r], prow[c2], a[r][c2]);
#pragma unroll
      for (int r = 0; r < RPL; ++r) a[r][CPW - 2] = w[r];
      const int p = pivot_row(kx);
      const R piv = __shfl_sync(FULL, vb, p & 31);
      const uint32_t ph = smem_u32(hs + (s & 1) * CPWP);
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const bool own = kr[r] == kx;
        msk[r] = own ? 0u : msk[r];
        cc[r] = own ? 0u : cc[r];
#pragma unroll
        for (int c2 = 0; c2 < CPW - 1; c2 += 2)
          st_pair_if(ph + c2 * sizeof(R), a[r][c2], c2 + 1 < CPW - 1 ? a[r][c2 + 1] : R(0), own);
      }
      __syncwarp();
      const R* hp = hs + (s & 1) * CPWP;
      R p0 = R(0);
#pragma unroll
      for (int c2 = 0; c2 < CPW - 1; c2 += 2) {
        const R2 v = reinterpret_cast<const R2*>(hp)[c2 / 2];
        if (c2 == 0)
          p0 = v.x;
        else
          prow[c2] = v.x;
        prow[c2 + 1] = v.y;
      }
      const R rp = rcp_rn(piv);
      if (piv == R(0)) st_local |= VB_STATUS_ZERO_PIVOT;
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const bool own = kr[r] == kx;
        m[r] = (own ? zero_as(t[r]) : t[r]) * rp;   // +0 on the pivot row
        w[r] = own ? R(1) : -m[r];
      }
#pragma unroll
      for (int r = 0; r < RPL; ++r) t[r] = fma(-m[r], p0, a[r][0]);
#pragma unroll
      for (int r = 0; r < RPL; ++r) Mq[s * NPR + lane + 32 * r] = m[r];
      pivs[k0 + s] = p;   // every lane stores the same values
      qs[p] = k0 + s;
      rps[p] = rp;
    }
#pragma unroll
    for (int c2 = 1; c2 < CPW - 1; ++c2)
#pragma unroll
      for (int r = 0; r < RPL; ++r) a[r][c2] = fma(-m[r], prow[c2], a[r][c2]);
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      a[r][0] = t[r];
      a[r][CPW - 1] = w[r];
    }
#pragma unroll 1
    for (int s = cnt; s < CPW; ++s) {   // a partial panel: finish the rotation
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const R t = a[r][0];
#pragma unroll
        for (int c2 = 1; c2 < CPW; ++c2) a[r][c2 - 1] = a[r][c2];
        a[r][CPW - 1] = t;
      }
    }
  };

  // Panel q's steps applied to this warp's columns, in order: the pivot row
  // of each step through the warp's hand-over slot (two by step parity).
  auto apply_panel = [&](int q) {
    const int k0 = q * CPW, cnt = min(CPW, n - k0);
    const R* Mq = Mb + (q & 1) * G::MS + lane;
    R* hs = Ub + warp * G::US;
#pragma unroll 3
    for (int s = 0; s < cnt; ++s) {
      const int p = pivs[k0 + s];
      R m[RPL], prow[CPWP];
#pragma unroll
      for (int r = 0; r < RPL; ++r) m[r] = Mq[s * NPR + 32 * r];
      const uint32_t ph = smem_u32(hs + (s & 1) * CPWP);
#pragma unroll
      for (int r = 0; r < RPL; ++r)
#pragma unroll
        for (int c2 = 0; c2 < CPWP; c2 += 2)
          st_pair_if(ph + c2 * sizeof(R), a[r][c2], c2 + 1 < CPW ? a[r][c2 + 1] : R(0), p == lane + 32 * r);
      __syncwarp();
#pragma unroll
      for (int c2 = 0; c2 < CPWP; c2 += 2) {
        const R2 v = reinterpret_cast<const R2*>(hs + (s & 1) * CPWP)[c2 / 2];
        prow[c2] = v.x;
        prow[c2 + 1] = v.y;
      }
#pragma unroll
      for (int c2 = 0; c2 < CPW; ++c2)
#pragma unroll
        for (int r = 0; r < RPL; ++r) a[r][c2] = fma(-m[r], prow[c2], a[r][c2]);
    }
    __syncwarp();
  };

  // Inv_j (in Ib) to global memory and the forward sweep of the right-hand
  // side, rhs[j+1] -= sub_d[j] o (Inv_j rhs[j]), by warps w0 .. NW-1.
  auto finish_layer = [&](int j, int w0) {
    {
      R2* O = reinterpret_cast<R2*>(out + (int64_t)j * iblk);
      const R2* S2 = reinterpret_cast<const R2*>(Ib);
      for (int e = (warp - w0) * 32 + lane; e < iblk / 2; e += (NW - w0) * 32) O[e] = S2[e];
    }
    if (!rhs || j + 1 >= nz) return;
    const double* cj = cpl + (j & 1) * 3 * NPR;
    const double* vc = vecs + (j & 1) * NPR;
    double* vn = vecs + ((j + 1) & 1) * NPR;
    // four lanes per row, eight rows per warp per pass (warp-uniform passes)
    const int sub = lane & 3;
    for (int i0 = (warp - w0) * 8; i0 < n; i0 += (NW - w0) * 8) {
      const int i = i0 + (lane >> 2);
      double s0 = 0.0, s1 = 0.0;
      if (i < n) {
        int m = sub;
        for (; m + 4 < n; m += 8) {
          s0 = fma((double)Ib[i * li + m], vc[m], s0);
          s1 = fma((double)Ib[i * li + m + 4], vc[m + 4], s1);
        }
        if (m < n) s0 = fma((double)Ib[i * li + m], vc[m], s0);
      }
      double s = s0 + s1;
      s += __shfl_xor_sync(FULL, s, 1);
      s += __shfl_xor_sync(FULL, s, 2);
      if (sub == 0 && i < n) {
        const double v = cj[2 * NPR + i] - cj[NPR + i] * s;
        rhs[(int64_t)(j + 1) * n + i] = v;
        vn[i] = v;
      }
    }
  };

  const int np = (n + CPW - 1) / CPW;   // panels holding columns of the block
  for (int j = 0; j < nz; ++j) {
    if (DPF) {
      const bool ok = mbar_wait(bar, (uint32_t)(j & 1), wlim);
      if (__syncthreads_or(!ok)) {
        // give up: wait (bounded) for the copy still in flight, report, return
        if (threadIdx.x == 0) {
          mbar_wait(bar, (uint32_t)(j & 1), WAIT_LIMIT);
          atomicOr(status, VB_STATUS_WATCHDOG);
        }
        return;
      }
    } else {
      __syncthreads();
    }
    // ---- D_j and the Hadamard Schur update from Inv_{j-1} (solver.py:47):
    //      tile element (i, m) = B[i][m], A'_j[m][i] when tr, else A'_j[i][m]
    {
      const double* D = DPF ? Db : Din + (int64_t)j * blk;
      const double* cp = cpl + ((j + 1) & 1) * 3 * NPR;   // of layer j-1
      double sr[RPL], sc[CPW];   // the sub_d / sup_d factor of tile row i and column m
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const int i = lane + 32 * r;
        sr[r] = (j > 0 && i < n) ? cp[(tr ? 0 : NPR) + i] : 0.0;
      }
#pragma unroll
      for (int c = 0; c < CPW; ++c) {
        const int m = warp * CPW + c;
        sc[c] = (j > 0 && m < n) ? cp[(tr ? NPR : 0) + m] : 0.0;
      }
      const int si = tr ? 1 : ld, sm = tr ? ld : 1;   // element strides of tile rows / columns in D
      const int ii = tr ? 1 : li, im = tr ? li : 1;   // and in Ib
      const double* rprev = rsc + ((j + 1) & 1) * NPC;
      double v[RPL][CPW];
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const int i = lane + 32 * r;
#pragma unroll
        for (int c = 0; c < CPW; ++c) {
          const int m = warp * CPW + c;
          double x = 0.0;
          if (i < n && m < n) {
            x = D[i * si + m * sm];
            if (j > 0) {
              const double cb = tr ? sc[c] * sr[r] : sr[r] * sc[c];
              double inv = (double)Ib[i * ii + m * im];
              if (EQ) inv = inv * rprev[i];
              x = x - cb * inv;
            }
          }
          v[r][c] = x;
        }
      }
      if (EQ) {
        // largest magnitude of each tile column (row m of A'_j): the column lives in this warp
        double* rcur = rsc + (j & 1) * NPC;
#pragma unroll
        for (int c = 0; c < CPW; ++c) {
          double cm = 0.0;
#pragma unroll
          for (int r = 0; r < RPL; ++r) cm = fmax(cm, fabs(v[r][c]));
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) cm = fmax(cm, __shfl_xor_sync(FULL, cm, off));
          const double s = pow2_scale(cm);
          const int m = warp * CPW + c;
          if (lane == 0 && m < n) {
            rcur[m] = s;
            rs_out[(int64_t)j * n + m] = s;
          }
#pragma unroll
          for (int r = 0; r < RPL; ++r) v[r][c] *= s;
        }
      }
#pragma unroll
      for (int r = 0; r < RPL; ++r)
#pragma unroll
        for (int c = 0; c < CPW; ++c) a[r][c] = (R)v[r][c];
    }
    for (int i = threadIdx.x; i < NPR; i += NW * 32) qs[i] = -1;
    __syncthreads();   // Db consumed, qs cleared
    if (j + 1 < nz) {
      if (DPF && threadIdx.x == 0) {
        fence_proxy_async();
        mbar_expect_tx(bar, dbytes);
        bulk_g2s(Db, Din + (int64_t)(j + 1) * blk, dbytes, bar);
      }
      // the coupling of layers j and j+1, for the next Schur update and the sweep
      if ((int)threadIdx.x < n) {
        double* cj = cpl + (j & 1) * 3 * NPR + threadIdx.x;
        cp_async8(cj, supn + (int64_t)j * n + threadIdx.x);
        cp_async8(cj + NPR, subn + (int64_t)j * n + threadIdx.x);
        if (rhs) cp_async8(cj + 2 * NPR, rhs + (int64_t)(j + 1) * n + threadIdx.x);
      }
    }
    // ---- elimination by panels; the other warps finish the previous layer
    //      while the first panel is eliminated
#pragma unroll 1
    for (int q = 0; q < np; ++q) {
      if (q == 0) {
        if (j > 0 && warp > 0) finish_layer(j - 1, 1);
      } else if (warp < np && warp != q - 1) {
        apply_panel(q - 1);
      }
      if (warp == q) factor_panel(q);
      __syncthreads();
    }
    if (warp < np - 1) apply_panel(np - 1);
    // ---- scale rows by 1/piv, scatter B^{-1}[q(i)][p_m] = T[i][m] into Ib
    //      (A'^{-1}[p_m][q(i)] when tr; q(i) = qs[i], the step pivoting on row i)
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int i = lane + 32 * r;
      if (i < n) {
        const R s = rps[i];
        const int qi = qs[i];
#pragma unroll
        for (int c = 0; c < CPW; ++c) {
          const int m = warp * CPW + c;
          if (m < n) {
            const R v = a[r][c] * s;
            if (!isfinite(v)) st_local |= VB_STATUS_NONFINITE;
            Ib[tr ? pivs[m] * li + qi : qi * li + pivs[m]] = v;
          }
        }
      }
    }
    cp_async_wait_all();
  }
  __syncthreads();
  finish_layer(nz - 1, 0);
  if (st_local) atomicOr(status, st_local);
}

// ---------------------------------------------------------------- FP64, trailing updates by DMMA
// D += A B for one m8n8k4 FP64 tile (A: 8x4 row, B: 4x8 col; per lane a =
// A[g][t], b = B[t][g], d = D[g][2t], D[g][2t+1], g = lane / 4, t = lane % 4).
// The unit adds the four products in the order k = 0..3 with one rounding
// each, so a tile equals the same four FMAs one after the other.
__device__ __forceinline__ void dmma_m8n8k4(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// Named barrier between two warps: the producer arrives, the consumer waits.
__device__ __forceinline__ void pair_arrive(int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void pair_wait(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

template <int NT>
struct DGJ {
  static constexpr int NP = 8 * NT;              // row and column capacity
  static constexpr int RPL = (NP + 31) / 32;     // rows per lane in the row layout
  static constexpr int MST = NP + 4;             // stride of a step's multipliers (4 or 12 mod 16: A fragments
                                                 // are read without bank conflicts)
  static constexpr int CST = 10;                 // row stride of the layout-change buffers
  static constexpr int XN = 2 * NT > 8 * RPL ? 2 * NT : 8 * RPL;
  __host__ __device__ static size_t al(size_t x) { return (x + 15) & ~(size_t)15; }
  static size_t smem_bytes(int n, int ld, bool dpf) {
    const size_t blk = (size_t)n * ld * sizeof(double);
    return al(blk)                                    // Ib: the inverse of the layer (natural order)
           + (dpf ? al(blk) : 0)                      // Db: the next diagonal block, prefetched
           + 6 * NP * sizeof(double)                  // cpl: sup_d[j], sub_d[j], rhs[j+1] (2 parities of j)
           + 2 * NP * sizeof(double)                  // vecs: right-hand side ping-pong
           + NP * sizeof(double)                      // rps: 1 / pivot of each row
           + 2 * 8 * MST * sizeof(double)             // Mb: multipliers of a panel's steps (2 parities)
           + 2 * 64 * sizeof(double)                  // Lb: multiplier of each step on the later pivot rows (2 par.)
           + NT * 64 * sizeof(double)                 // Ub: pivot rows, a block per warp
           + 2 * NP * CST * sizeof(double)            // Cv: layout changes (to rows, to fragments)
           + 2 * NP * sizeof(int)                     // pivs, qs: pivot row of each step, step of each row (-1: none)
           + 16;                                      // mbarrier of the prefetch
  }
};

// The same factor in FP64 (panel_factor_atmosphere says what is computed and
// why), with the trailing updates on the FP64 tensor cores. One warp per panel
// of 8 columns:
//  * Warp q runs panel q's 8 pivot steps alone, from registers, in the row
//    layout; the warp of panel q + 1 follows it step by step (a named barrier
//    per step, producer side not blocking), so the next panel starts a step
//    after this one ends; every other warp applies the panel as a whole,
//    S[:, C] -= M U, one block barrier per panel instead of one per step.
//  * A panel is applied four steps at a time by mma.sync m8n8k4: the operands
//    arrive as fragments, 1 double per lane for 8 FMAs. With the pivot row and
//    the multipliers broadcast to every lane (the scalar form) the loads, not
//    the FMAs, filled the time: a step moved 24 KB through shared memory at
//    69 columns. The DMMA adds its four products in step order with one
//    rounding each, so every element sees the FMAs of the scalar elimination
//    in the same order: the results are the scalar kernels' bit for bit.
//  * The first right-hand side's sweep of the layer before and the store of
//    its inverse run in the idle warps while the first panel is eliminated.
// Bound by the chain of pivot steps: about 270 cycles a step alone (150
// instructions of one warp, issued in order), 370 beside the other warps of
// the block, 600 with two blocks on the SM. Factor of nz=120, ni=69 (B200, ms,
// one block barrier per step before, this kernel now): one atmosphere 3.07,
// 2.12 (34.7K cycles a layer); 148 (one per SM) 3.21, 2.13; 296 (two per SM)
// 5.64, 3.70; ni=89, nz=150, 128 atmospheres 6.03, 4.12; ni=30, nz=43, one 0.349,
// 0.242.
// WIDE: registers for both halves of a panel's update at once (one block on the
// SM).
template <int NT, bool DPF, bool WIDE>
__device__ __forceinline__ void dmma_factor_atmosphere(int nz, int n, int ld, const double* Din, double* out,
                                                       const double* __restrict__ supn,
                                                       const double* __restrict__ subn, double* rhs, bool tr,
                                                       int32_t* status, char* smem_raw, long long wlim) {
  using G = DGJ<NT>;
  constexpr int NP = G::NP, RPL = G::RPL, MST = G::MST, CST = G::CST, NW = NT;
  static_assert(NT >= 3, "two warps eliminate the first panel while the others finish the previous layer");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const unsigned FULL = 0xffffffffu;
  const int blk = n * ld;
  char* sp = smem_raw;
  auto take = [&](size_t bytes) {
    char* q = sp;
    sp += G::al(bytes);
    return q;
  };
  double* Ib = reinterpret_cast<double*>(take((size_t)blk * sizeof(double)));
  double* Db = DPF ? reinterpret_cast<double*>(take((size_t)blk * sizeof(double))) : nullptr;
  double* cpl = reinterpret_cast<double*>(take(6 * NP * sizeof(double)));
  double* vecs = reinterpret_cast<double*>(take(2 * NP * sizeof(double)));
  double* rps = reinterpret_cast<double*>(take(NP * sizeof(double)));
  double* Mb = reinterpret_cast<double*>(take(2 * 8 * MST * sizeof(double)));
  double* Lb = reinterpret_cast<double*>(take(2 * 64 * sizeof(double)));
  double* Uw = reinterpret_cast<double*>(take(NT * 64 * sizeof(double))) + warp * 64;
  double* Cv = reinterpret_cast<double*>(take(2 * NP * CST * sizeof(double)));
  int* pivs = reinterpret_cast<int*>(take(NP * sizeof(int)));
  int* qs = reinterpret_cast<int*>(take(NP * sizeof(int)));
  uint64_t* bar = reinterpret_cast<uint64_t*>(take(16));
  const uint32_t dbytes = (uint32_t)(blk * sizeof(double));
  int st_local = 0;

  for (int e = threadIdx.x; e < blk; e += NW * 32) Ib[e] = 0.0;   // the padding columns stay 0
  if (rhs)
    for (int i = threadIdx.x; i < n; i += NW * 32) vecs[i] = rhs[i];
  if (DPF && threadIdx.x == 0) mbar_init(bar, 1);
  __syncthreads();
  if (DPF && threadIdx.x == 0) {
    mbar_expect_tx(bar, dbytes);
    bulk_g2s(Db, Din, dbytes, bar);
  }

  // The warp's 8 columns, in one of two layouts sharing the registers:
  //   fragments  XF(a, e): row 8 a + g, column 2 t4 + e (mma accumulators)
  //   rows       XR(r, c): row lane + 32 r, column c
  double x[G::XN];
#define XF(a, e) x[2 * (a) + (e)]
#define XR(r, c) x[8 * (r) + (c)]
  // key of row r: magnitude under msk above cc; both 0 for rows that may not pivot
  unsigned msk[RPL], cc[RPL];

  auto to_rows = [&]() {
    double* C = Cv;
#pragma unroll
    for (int a = 0; a < NT; ++a)
      *reinterpret_cast<double2*>(C + (8 * a + g) * CST + 2 * t4) = double2{XF(a, 0), XF(a, 1)};
    __syncwarp();
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int i = lane + 32 * r;
      const bool in = 32 * r + 31 < NP || i < NP;
#pragma unroll
      for (int c = 0; c < 8; c += 2) {
        double2 v = double2{0.0, 0.0};
        if (in) v = *reinterpret_cast<const double2*>(C + i * CST + c);
        XR(r, c) = v.x;
        XR(r, c + 1) = v.y;
      }
    }
  };
  auto to_frags = [&]() {
    double* C = Cv + NP * CST;
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int i = lane + 32 * r;
      if (32 * r + 31 < NP || i < NP)
#pragma unroll
        for (int c = 0; c < 8; c += 2)
          *reinterpret_cast<double2*>(C + i * CST + c) = double2{XR(r, c), XR(r, c + 1)};
    }
    __syncwarp();
#pragma unroll
    for (int a = 0; a < NT; ++a) {
      const double2 v = *reinterpret_cast<const double2*>(C + (8 * a + g) * CST + 2 * t4);
      XF(a, 0) = v.x;
      XF(a, 1) = v.y;
    }
  };

  // The pivot steps of panel q (columns 8 q + s), run by the warp that owns
  // them (row layout).
  auto factor_panel = [&](int q, bool followed) {
    const int k0 = q * 8, cnt = min(8, n - k0);
    double* Mq = Mb + (q & 1) * 8 * MST;
    double* Lq = Lb + (q & 1) * 64;
    const int ll = min(lane, 7);
    double lv = 0.0;
#pragma unroll 1
    for (int s = 0; s < cnt; ++s) {
      unsigned kr[RPL];
#pragma unroll
      for (int r = 0; r < RPL; ++r) kr[r] = (pivot_mag(XR(r, 0)) & msk[r]) | cc[r];
      const unsigned km = key_max(kr);
      const unsigned kx = __reduce_max_sync(FULL, km);
      double vb = XR(0, 0);   // this lane's candidate
#pragma unroll
      for (int r = 1; r < RPL; ++r) vb = kr[r] == km ? XR(r, 0) : vb;
      const int p = pivot_row(kx);
      const double piv = __shfl_sync(FULL, vb, p & 31);
      const uint32_t ph = smem_u32(Uw + (s & 1) * 8);
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const bool own = kr[r] == kx;
        msk[r] = own ? 0u : msk[r];
        cc[r] = own ? 0u : cc[r];
#pragma unroll
        for (int c = 0; c < 8; c += 2) st_pair_if(ph + c * sizeof(double), XR(r, c), XR(r, c + 1), own);
      }
      __syncwarp();
      const double2* hp = reinterpret_cast<const double2*>(Uw + (s & 1) * 8);
      const double2 h0 = hp[0], h1 = hp[1], h2 = hp[2], h3 = hp[3];
      const double rp = rcp_rn(piv);
      if (piv == 0.0) st_local |= VB_STATUS_ZERO_PIVOT;
      double m[RPL];
#pragma unroll
      for (int r = 0; r < RPL; ++r) m[r] = (kr[r] == kx ? zero_as(XR(r, 0)) : XR(r, 0)) * rp;   // +0 on the pivot row
#pragma unroll
      for (int r = 0; r < RPL; ++r) XR(r, 0) = fma(-m[r], h0.y, XR(r, 1));
#pragma unroll
      for (int r = 0; r < RPL; ++r)
        if (32 * r + 31 < NP || lane + 32 * r < NP) Mq[s * MST + lane + 32 * r] = m[r];
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        XR(r, 1) = fma(-m[r], h1.x, XR(r, 2));
        XR(r, 2) = fma(-m[r], h1.y, XR(r, 3));
        XR(r, 3) = fma(-m[r], h2.x, XR(r, 4));
        XR(r, 4) = fma(-m[r], h2.y, XR(r, 5));
        XR(r, 5) = fma(-m[r], h3.x, XR(r, 6));
        XR(r, 6) = fma(-m[r], h3.y, XR(r, 7));
        XR(r, 7) = kr[r] == kx ? 1.0 : -m[r];   // the step's finished column
      }
      pivs[k0 + s] = p;   // every lane stores the same values
      qs[p] = k0 + s;
      rps[p] = rp;
      if (followed) pair_arrive(1 + s);
      if (s > 0) Lq[ll * 8 + s - 1] = lv;
      lv = Mq[ll * MST + p];
    }
    Lq[ll * 8 + cnt - 1] = lv;
#pragma unroll 1
    for (int s = cnt; s < 8; ++s) {   // a partial panel: finish the rotation, no multipliers
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const double v = XR(r, 0);
#pragma unroll
        for (int c = 1; c < 8; ++c) XR(r, c - 1) = XR(r, c);
        XR(r, 7) = v;
        if (32 * r + 31 < NP || lane + 32 * r < NP) Mq[s * MST + lane + 32 * r] = 0.0;
      }
    }
  };

  // The next panel's warp takes panel q's steps one by one as they are
  // published (row layout), a step or two behind their owner.
  auto follow_panel = [&](int q) {
    const int k0 = q * 8;   // a full panel: the next one holds columns
    const double* Mq = Mb + (q & 1) * 8 * MST;
#pragma unroll 1
    for (int s = 0; s < 8; ++s) {
      pair_wait(1 + s);
      const int p = pivs[k0 + s];
      double m[RPL];
#pragma unroll
      for (int r = 0; r < RPL; ++r)
        m[r] = (32 * r + 31 < NP || lane + 32 * r < NP) ? Mq[s * MST + lane + 32 * r] : 0.0;
      const uint32_t ph = smem_u32(Uw + (s & 1) * 8);
#pragma unroll
      for (int r = 0; r < RPL; ++r) {
        const bool own = p == lane + 32 * r;
        msk[r] = own ? 0u : msk[r];
        cc[r] = own ? 0u : cc[r];
#pragma unroll
        for (int c = 0; c < 8; c += 2) st_pair_if(ph + c * sizeof(double), XR(r, c), XR(r, c + 1), own);
      }
      __syncwarp();
      const double2* hp = reinterpret_cast<const double2*>(Uw + (s & 1) * 8);
#pragma unroll
      for (int c = 0; c < 8; c += 2) {
        const double2 h = hp[c / 2];
#pragma unroll
        for (int r = 0; r < RPL; ++r) {
          XR(r, c) = fma(-m[r], h.x, XR(r, c));
          XR(r, c + 1) = fma(-m[r], h.y, XR(r, c + 1));
        }
      }
    }
  };

  // Panel q's steps on this warp's columns (fragments), four at a time: the
  // four pivot rows are gathered, brought to their state at their own step
  // (lane (g, t4) forms column g) and every row then takes the four steps in
  // one DMMA per tile. Each element sees the same FMAs in the same order as
  // step by step.
  auto apply_panel = [&](int q) {
    const int k0 = q * 8, cnt = min(8, n - k0);
    const double* Mq = Mb + (q & 1) * 8 * MST;
    const double* Lq = Lb + (q & 1) * 64;
    int sl[NT];   // the panel's step of each row (others out of 0..7)
#pragma unroll
    for (int a = 0; a < NT; ++a) sl[a] = qs[8 * a + g] - k0;
#pragma unroll(WIDE ? 2 : 1)
    for (int h = 0; h < 2; ++h) {
      double* U = Uw + 32 * h;
      const uint32_t us = smem_u32(Uw + 2 * t4);
      const double2 l01 = *reinterpret_cast<const double2*>(Lq + (4 * h) * 8 + 4 * h);       // .y: step 0 on row 1
      const double2 l02 = *reinterpret_cast<const double2*>(Lq + (4 * h) * 8 + 4 * h + 2);   // step 0 on rows 2, 3
      const double2 l12 = *reinterpret_cast<const double2*>(Lq + (4 * h + 1) * 8 + 4 * h + 2);
      const double l23 = Lq[(4 * h + 2) * 8 + 4 * h + 3];
#pragma unroll
      for (int a = 0; a < NT; ++a) st_pair_if(us + sl[a] * 64, XF(a, 0), XF(a, 1), (unsigned)(sl[a] - 4 * h) < 4u);
      __syncwarp();
      double u0 = U[g], u1 = U[8 + g], u2 = U[16 + g], u3 = U[24 + g];
      // steps past a partial panel's end: zero multipliers and zero rows
      if (4 * h >= cnt) u0 = 0.0;
      u1 = 4 * h + 1 >= cnt ? 0.0 : fma(-l01.y, u0, u1);
      u2 = 4 * h + 2 >= cnt ? 0.0 : fma(-l12.x, u1, fma(-l02.x, u0, u2));
      u3 = 4 * h + 3 >= cnt ? 0.0 : fma(-l23, u2, fma(-l12.y, u1, fma(-l02.y, u0, u3)));
      const double b = -(t4 < 2 ? (t4 == 0 ? u0 : u1) : (t4 == 2 ? u2 : u3));
      const double* Ma = Mq + (4 * h + t4) * MST + g;
#pragma unroll
      for (int a = 0; a < NT; ++a) dmma_m8n8k4(XF(a, 0), XF(a, 1), Ma[8 * a], b);
    }
  };

  // Inv_j (in Ib) to global memory and the forward sweep of the right-hand
  // side, rhs[j+1] -= sub_d[j] o (Inv_j rhs[j]), by warps w0 .. NW-1.
  auto finish_layer = [&](int j, int w0) {
    {
      double2* O = reinterpret_cast<double2*>(out + (int64_t)j * blk);
      const double2* S2 = reinterpret_cast<const double2*>(Ib);
#pragma unroll 4
      for (int e = (warp - w0) * 32 + lane; e < blk / 2; e += (NW - w0) * 32) O[e] = S2[e];
    }
    if (!rhs || j + 1 >= nz) return;
    const double* cj = cpl + (j & 1) * 3 * NP;
    const double* vc = vecs + (j & 1) * NP;
    double* vn = vecs + ((j + 1) & 1) * NP;
    // four lanes per row, eight rows per warp per pass (warp-uniform passes), the
    // rows dealt against bank conflicts as in the sweeps
    const int sub = lane & 3;
    for (int i0 = (warp - w0) * 8; i0 < n; i0 += (NW - w0) * 8) {
      const int i = i0 + ((2 * g) & 7) + (g >> 2);
      const double* row = Ib + min(i, n - 1) * ld;
      double s0 = 0.0, s1 = 0.0;
      int m = sub;
#pragma unroll 4
      for (; m + 4 < n; m += 8) {
        s0 = fma(row[m], vc[m], s0);
        s1 = fma(row[m + 4], vc[m + 4], s1);
      }
      if (m < n) s0 = fma(row[m], vc[m], s0);
      double s = s0 + s1;
      s += __shfl_xor_sync(FULL, s, 1);
      s += __shfl_xor_sync(FULL, s, 2);
      if (sub == 0 && i < n) {
        const double v = cj[2 * NP + i] - cj[NP + i] * s;
        rhs[(int64_t)(j + 1) * n + i] = v;
        vn[i] = v;
      }
    }
  };

  const int np = (n + 7) >> 3;   // panels holding columns of the block
  for (int j = 0; j < nz; ++j) {
    if (DPF) {
      const bool ok = mbar_wait(bar, (uint32_t)(j & 1), wlim);
      if (__syncthreads_or(!ok)) {
        // give up: wait (bounded) for the copy still in flight, report, return
        if (threadIdx.x == 0) {
          mbar_wait(bar, (uint32_t)(j & 1), WAIT_LIMIT);
          atomicOr(status, VB_STATUS_WATCHDOG);
        }
        return;
      }
    } else {
      __syncthreads();
    }
    // ---- D_j and the Hadamard Schur update from Inv_{j-1} (solver.py:47):
    //      tile element (i, m) = B[i][m], A'_j[m][i] when tr, else A'_j[i][m]
    {
      const double* D = DPF ? Db : Din + (int64_t)j * blk;
      const double* cp = cpl + ((j + 1) & 1) * 3 * NP;   // of layer j-1
      const double* cr = cp + (tr ? 0 : NP);             // the sub_d / sup_d factor of tile row i
      const double* cm = cp + (tr ? NP : 0);             // and column m
      const int si = tr ? 1 : ld, sm = tr ? ld : 1;      // element strides of tile rows / columns in D and Ib
      // element at offset o with the coupling factors f (sup_d sub_d of row and column)
      auto element = [&](bool in, int o, double f) {
        double v = in ? D[o] : 0.0;
        if (j > 0 && in) v = v - f * Ib[o];
        return v;
      };
      if (warp < 2) {
        double f[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) f[c] = 8 * warp + c < n ? cm[8 * warp + c] : 0.0;
#pragma unroll
        for (int r = 0; r < RPL; ++r) {
          const int i = lane + 32 * r;
          const double fr = i < n ? cr[i] : 0.0;
#pragma unroll
          for (int c = 0; c < 8; ++c)
            XR(r, c) = element(i < n && 8 * warp + c < n, i * si + (8 * warp + c) * sm, f[c] * fr);
          msk[r] = i < n ? 0xffffff00u : 0u;
          cc[r] = i < n ? 255u - (unsigned)i : 0u;
        }
      } else {
        const int m = 8 * warp + 2 * t4;
        const double f0 = m < n ? cm[m] : 0.0, f1 = m + 1 < n ? cm[m + 1] : 0.0;
#pragma unroll
        for (int a = 0; a < NT; ++a) {
          const int i = 8 * a + g;
          const double fr = i < n ? cr[i] : 0.0;
          XF(a, 0) = element(i < n && m < n, i * si + m * sm, f0 * fr);
          XF(a, 1) = element(i < n && m + 1 < n, i * si + (m + 1) * sm, f1 * fr);
        }
      }
    }
    for (int i = threadIdx.x; i < NP; i += NW * 32) qs[i] = -1;
    __syncthreads();   // Db consumed, qs cleared
    if (j + 1 < nz) {
      if (DPF && threadIdx.x == 0) {
        fence_proxy_async();
        mbar_expect_tx(bar, dbytes);
        bulk_g2s(Db, Din + (int64_t)(j + 1) * blk, dbytes, bar);
      }
      // the coupling of layers j and j+1, for the next Schur update and the sweep
      if ((int)threadIdx.x < n) {
        double* cj = cpl + (j & 1) * 3 * NP + threadIdx.x;
        cp_async8(cj, supn + (int64_t)j * n + threadIdx.x);
        cp_async8(cj + NP, subn + (int64_t)j * n + threadIdx.x);
        if (rhs) cp_async8(cj + 2 * NP, rhs + (int64_t)(j + 1) * n + threadIdx.x);
      }
    }
    // ---- elimination by panels
#pragma unroll 1
    for (int q = 0; q < np; ++q) {
      if (warp == q) {
        factor_panel(q, q + 1 < np);
      } else if (warp == q + 1 && q + 1 < np) {
        if (q > 0) {
#pragma unroll
          for (int r = 0; r < RPL; ++r) {   // rows left by the panels before q
            const int i = lane + 32 * r;
            const bool fr = i < n && qs[i] < 0;
            msk[r] = fr ? 0xffffff00u : 0u;
            cc[r] = fr ? 255u - (unsigned)i : 0u;
          }
          apply_panel(q - 1);
          to_rows();
        }
        follow_panel(q);
      } else if (q == 0) {
        if (j > 0 && warp >= 2) finish_layer(j - 1, 2);
      } else if (warp == q - 1) {
        to_frags();
      } else if (warp < np) {
        apply_panel(q - 1);
      }
      __syncthreads();
    }
    if (warp < np - 1)
      apply_panel(np - 1);
    else if (warp == np - 1)
      to_frags();
    // ---- scale rows by 1/piv, scatter B^{-1}[q(i)][p_m] = T[i][m] into Ib
    //      (A'^{-1}[p_m][q(i)] when tr; q(i) = qs[i], the step pivoting on row i)
    if (warp < np) {
      const int m = 8 * warp + 2 * t4;
      const int qstr = tr ? 1 : ld, pstr = tr ? ld : 1;
      const bool on0 = m < n, on1 = m + 1 < n;
      double* d0 = Ib + (on0 ? pivs[m] * pstr : 0);
      double* d1 = Ib + (on1 ? pivs[m + 1] * pstr : 0);
      unsigned top = 0;   // largest exponent field of the results: all ones when not finite
#pragma unroll
      for (int a = 0; a < NT; ++a) {
        const int i = 8 * a + g;
        if (i < n) {
          const double s = rps[i], v0 = XF(a, 0) * s, v1 = XF(a, 1) * s;
          const int at = qs[i] * qstr;
          if (on0) {
            d0[at] = v0;
            top = max(top, (unsigned)__double2hiint(v0) & 0x7ff00000u);
          }
          if (on1) {
            d1[at] = v1;
            top = max(top, (unsigned)__double2hiint(v1) & 0x7ff00000u);
          }
        }
      }
      if (top == 0x7ff00000u) st_local |= VB_STATUS_NONFINITE;
    }
    cp_async_wait_all();
  }
  __syncthreads();
  finish_layer(nz - 1, 0);
  if (st_local) atomicOr(status, st_local);
#undef XF
#undef XR
}

}  // namespace vb
