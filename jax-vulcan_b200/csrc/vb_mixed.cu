// Mixed-precision block-tridiagonal solve: the diagonal blocks are factored
// and inverted in FP32 (same kernel as the FP64 path, element type float),
// and the solution is recovered in FP64 by iterative refinement on the full
// block-tridiagonal system
//     r = b - M x          (FP64, from the FP64 blocks and off-diagonals)
//     x = x + M~^{-1} r     (block-Thomas sweeps with the FP32 inverses)
// until max|correction| <= tol * max|x|. Atmospheres whose refinement stalls
// are refactored and solved in FP64 and flagged VB_STATUS_REFINE_STALL.
// M is the system of reference solver.py:33-112: diagonal blocks A_j,
// sub-diagonal diag(sub_d[j-1]) at (j, j-1), super-diagonal diag(sup_d[j])
// at (j, j+1).
#include <cuda_runtime.h>

#include "vb_common.cuh"
#include "vb_launch.cuh"
#include "vb_sweep.cuh"

namespace vb {

constexpr int REFINE_THREADS = 256;
constexpr int REFINE_WARPS = REFINE_THREADS / 32;

// y[i] = sum_m A[i][m] (sc[m] v[m]) for an n x n block of row stride ld (one
// warp per row, lanes over columns; sc = nullptr: no column scales); v and y
// in shared memory.
template <typename T>
__device__ inline void block_mv(const T* __restrict__ A, int n, int ld, const double* v, double* y,
                                const double* __restrict__ sc = nullptr) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = warp; i < n; i += REFINE_WARPS) {
    double s = 0.0;
    for (int m = lane; m < n; m += 32) s = fma((double)A[(int64_t)i * ld + m], sc ? sc[m] * v[m] : v[m], s);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) y[i] = s;
  }
}

// One pass of refinement for every atmosphere (CTA per atmosphere). first:
// x is taken as 0 (the pass is the plain solve). state[b]: 1 once converged
// (later passes skip it). only != nullptr: atmospheres with only[b] == 0 skip.
// The inverses: inv (stride ld), or with mxr != nullptr (R = float) the
// row-equilibrated factors of the mixed region, A'_j^{-1} = X_j diag(r_j).
template <typename R>
__global__ void __launch_bounds__(REFINE_THREADS)
refine_kernel(Batch B, double* __restrict__ ws, const R* __restrict__ inv, const void* __restrict__ mxr,
              const double* __restrict__ rhs, double* __restrict__ x, int32_t* __restrict__ state,
              int32_t* __restrict__ passes, double tol, int first, const int32_t* __restrict__ only) {
  __shared__ double sx[VB_MAX_NI], sv[VB_MAX_NI], sr[VB_MAX_NI], su[VB_MAX_NI];
  __shared__ double red[REFINE_WARPS][2];
  const int b = blockIdx.x;
  if (only && only[b] == 0) return;
  if (!first && state[b] == 1) return;
  const Geo g = geo_of(B, b);
  const int n = B.ni, nz = g.nz, ld = B.ld;
  WsView w = ws_view(ws, g, n, ld);
  const R* Ib = inv + g.z0 * n * ld;
  int li = ld;                    // row stride of the inverses
  const double* rsc = nullptr;    // their column scales [nz][ni], if equilibrated
  if (mxr) {
    const MxView m = mx_view(const_cast<void*>(mxr), g.z0, nz, n);
    Ib = reinterpret_cast<const R*>(m.X);
    rsc = m.rs;
    li = round4(n);
  }
  const double* bb = rhs + g.z0 * n;
  double* xb = x + g.z0 * n;
  double* rp = w.rmod;   // forward-eliminated residual, [nz][ni]
  // ---- forward: r_j = b_j - (M x)_j, r'_j = r_j - sub[j-1] o (Inv_{j-1} r'_{j-1})
  for (int j = 0; j < nz; ++j) {
    if (!first)
      for (int i = threadIdx.x; i < n; i += blockDim.x) sx[i] = xb[(int64_t)j * n + i];
    __syncthreads();
    if (!first) block_mv(w.inv + (int64_t)j * n * ld, n, ld, sx, su);   // A_j x_j (FP64 blocks)
    if (j > 0)                                                           // Inv_{j-1} r'_{j-1}
      block_mv(Ib + (int64_t)(j - 1) * n * li, n, li, sr, sv, rsc ? rsc + (int64_t)(j - 1) * n : nullptr);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      double r = bb[(int64_t)j * n + i];
      if (!first) {
        double mx = su[i];
        if (j > 0) mx = mx + w.subn[(int64_t)(j - 1) * n + i] * xb[(int64_t)(j - 1) * n + i];
        if (j < nz - 1) mx = mx + w.supn[(int64_t)j * n + i] * xb[(int64_t)(j + 1) * n + i];
        r = r - mx;
      }
      if (j > 0) r = r - w.subn[(int64_t)(j - 1) * n + i] * sv[i];
      rp[(int64_t)j * n + i] = r;
      sr[i] = r;
    }
    __syncthreads();
  }
  // ---- backward: c_j = Inv_j (r'_j - sup[j] o c_{j+1}); x_j += c_j
  double cmax = 0.0, xmax = 0.0;
  for (int j = nz - 1; j >= 0; --j) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      double v = rp[(int64_t)j * n + i];
      if (j < nz - 1) v = v - w.supn[(int64_t)j * n + i] * su[i];
      sv[i] = v;
    }
    __syncthreads();
    block_mv(Ib + (int64_t)j * n * li, n, li, sv, sr, rsc ? rsc + (int64_t)j * n : nullptr);   // c_j
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const double c = sr[i];
      const double xn = (first ? 0.0 : xb[(int64_t)j * n + i]) + c;
      xb[(int64_t)j * n + i] = xn;
      su[i] = c;
      cmax = fmax(cmax, fabs(c));
      xmax = fmax(xmax, fabs(xn));
      if (!isfinite(xn)) cmax = INFINITY;
    }
    __syncthreads();
  }
  // ---- convergence of this atmosphere
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    cmax = fmax(cmax, __shfl_xor_sync(0xffffffffu, cmax, off));
    xmax = fmax(xmax, __shfl_xor_sync(0xffffffffu, xmax, off));
  }
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5][0] = cmax;
    red[threadIdx.x >> 5][1] = xmax;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double cm = red[0][0], xm = red[0][1];
    for (int q = 1; q < REFINE_WARPS; ++q) {
      cm = fmax(cm, red[q][0]);
      xm = fmax(xm, red[q][1]);
    }
    passes[b] += 1;
    // the first pass is the plain solve; its correction is x itself
    state[b] = (!first && cm <= tol * xm) ? 1 : 0;
  }
}

// After the FP32 passes: atmospheres that did not converge get the FP64
// fallback (fallback[b] = 1) and VB_STATUS_REFINE_STALL.
__global__ void refine_finalize_kernel(int batch, const int32_t* __restrict__ state, int32_t* __restrict__ fallback,
                                       int32_t* __restrict__ status) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  const int f = state[b] == 1 ? 0 : 1;
  fallback[b] = f;
  if (f) status[b] |= VB_STATUS_REFINE_STALL;
}

template <typename R>
cudaError_t launch_refine(const Batch& B, double* ws, const R* inv, const void* mxr, const double* rhs, double* x,
                          int32_t* state, int32_t* passes, double tol, int first, const int32_t* only,
                          cudaStream_t st) {
  refine_kernel<R><<<B.count, REFINE_THREADS, 0, st>>>(B, ws, inv, mxr, rhs, x, state, passes, tol, first, only);
  return cudaGetLastError();
}
template cudaError_t launch_refine<float>(const Batch&, double*, const float*, const void*, const double*, double*,
                                          int32_t*, int32_t*, double, int, const int32_t*, cudaStream_t);
template cudaError_t launch_refine<double>(const Batch&, double*, const double*, const void*, const double*, double*,
                                           int32_t*, int32_t*, double, int, const int32_t*, cudaStream_t);

cudaError_t launch_refine_finalize(int batch, const int32_t* state, int32_t* fallback, int32_t* status,
                                   cudaStream_t st) {
  refine_finalize_kernel<<<(batch + 127) / 128, 128, 0, st>>>(batch, state, fallback, status);
  return cudaGetLastError();
}

// ================================================================ mixed-precision Ros2 step
// Modes of an atmosphere (mode[b]) during the solves of one step:
//   MX_REFINE  FP32 inverses, refinement still running for this right-hand side
//   MX_DONE    FP32 inverses, refinement converged for this right-hand side
//   MX_FP64    FP64 inverses in place of its blocks (the FP32 factor failed or
//              refinement stalled): solved directly, no refinement
enum MxMode { MX_REFINE = 0, MX_DONE = 1, MX_FP64 = 3 };

__host__ __device__ inline size_t mx_al(size_t x) { return (x + 127) & ~(size_t)127; }
// Bytes of one ring stage: one inverse (FP32 X_j, or the FP64 inverse of an
// atmosphere in MX_FP64, which is the larger). The ring is sized in FP64
// stages; an FP32 atmosphere cuts it into as many of its own.
__host__ __device__ inline size_t mx_stage_bytes(int ni, bool f64) {
  return mx_al(f64 ? (size_t)ni * round_even(ni) * 8 : (size_t)ni * round4(ni) * 4);
}
__host__ __device__ inline size_t mx_pass_smem(int ni, int stages) {
  return stages * mx_stage_bytes(ni, true) + 64 + 2 * VB_MAX_NI * sizeof(double);
}

// A pass of the mixed-precision block solve of every atmosphere, right-hand
// side b = the workspace's rmod rows, solution x = its k1 rows (xsel 0) or aux
// rows (xsel 1).
//  first: x = M~^{-1} b with the factor's inverses (FP32 X_j with row scales,
//         or FP64 for MX_FP64 atmospheres); MX_DONE atmospheres restart as
//         MX_REFINE (a new right-hand side).
//  else:  MX_REFINE atmospheres: r = b - M x with the FP64 blocks D_j and
//         off-diagonals (the system of reference solver.py:33-112),
//         x += M~^{-1} r; MX_DONE once max|correction| <= tol max|x|.
// The residual's layers are independent: mx_residual_kernel forms them with a
// CTA per layer, straight from HBM, ahead of the sweeps (mx_sweep_kernel), whose
// chain then holds the FP32 inverses only (vb_sweep.cuh's form). With both in
// one kernel, a layer's residual on the chain and four barriers a layer, a
// refinement pass of 148 atmospheres (ni=69, nz=120) took 0.68 ms and a first
// pass 0.27; the residual now takes 0.08, the sweeps of either 0.26.

// Residual rows r_j = b_j - (M x)_j of the refining atmospheres into mv.tmp.
template <int N8>
__global__ void __launch_bounds__(32 * N8)
mx_residual_kernel(Batch B, double* __restrict__ ws, void* __restrict__ mxr, int xsel,
                   const int32_t* __restrict__ mode, const int32_t* __restrict__ only) {
  __shared__ double x0[VB_MAX_NI];
  const int b = blockIdx.y, j = blockIdx.x;
  if ((only && only[b] == 0) || mode[b] != MX_REFINE) return;
  const Geo g = geo_of(B, b);
  const int n = B.ni, nz = g.nz, ld = B.ld;
  if (j >= nz) return;
  WsView w = ws_view(ws, g, n, ld);
  MxView mv = mx_view(mxr, g.z0, nz, n);
  const double* xb = (xsel ? w.aux : w.k1) + (int64_t)j * n;
  for (int i = threadIdx.x; i < n; i += 32 * N8) x0[i] = xb[i];
  __syncthreads();
  const int row = sweep_row();
  const double p = row_dot<N8>(w.inv + (int64_t)j * n * ld, n, ld, row, x0);
  if (row < n && (threadIdx.x & 3) == 0) {
    const int64_t at = (int64_t)j * n + row;
    double mx = p;
    if (j > 0) mx = mx + w.subn[at - n] * xb[row - n];
    if (j < nz - 1) mx = mx + w.supn[at] * xb[row + n];
    mv.tmp[at] = w.rmod[at] - mx;
  }
}

// The sweeps of one atmosphere: forward r'_j = r_j - sub[j-1] o (Inv_{j-1}
// r'_{j-1}) (r: b on the first pass, else the residual rows) into mv.tmp,
// backward c_j = Inv_j (r'_j - sup[j] o c_{j+1}), x_j += c_j (x_j = c_j on the
// first pass). Blocks Inv_0 .. Inv_{nz-2}, then Inv_{nz-1} .. Inv_0, as one
// stream; N8 = ceil(ni / 8) warps of rows and one that copies.
template <int N8>
__global__ void __launch_bounds__(32 * N8 + 32)
mx_sweep_kernel(Batch B, double* __restrict__ ws, void* __restrict__ mxr, int xsel, int first,
                int32_t* __restrict__ mode, const int32_t* __restrict__ only, int32_t* __restrict__ passes, double tol,
                int32_t* __restrict__ status, int stages64, long long wlim) {
  extern __shared__ __align__(128) char smem_raw[];
  __shared__ double red[N8][2];
  __shared__ int redb[N8];
  const int b = blockIdx.x;
  if (only && only[b] == 0) return;
  const int md = mode[b];
  if (!first && md != MX_REFINE) return;
  const bool f64 = md == MX_FP64;
  const Geo g = geo_of(B, b);
  const int n = B.ni, nz = g.nz, ld = B.ld, ldf = round4(n);
  WsView w = ws_view(ws, g, n, ld);
  MxView mv = mx_view(mxr, g.z0, nz, n);
  double* xb = xsel ? w.aux : w.k1;
  const uint32_t bytes = f64 ? (uint32_t)(n * ld * 8) : (uint32_t)(n * ldf * 4);
  const size_t sb = mx_stage_bytes(n, f64), ring = stages64 * mx_stage_bytes(n, true);
  const int stages = min(SWEEP_MAX_STAGES, (int)(ring / sb));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + ring);
  double* v = reinterpret_cast<double*>(bars + 8);   // [2][VB_MAX_NI]: the (scaled) operand, by step parity
  const int F = nz - 1, count = F + nz;              // forward blocks, all blocks
  auto src = [&](int s) -> const void* {
    const int64_t j = s < F ? s : count - 1 - s;
    return f64 ? static_cast<const void*>(w.inv + j * n * ld) : static_cast<const void*>(mv.X + j * n * ldf);
  };
  BlockStream<decltype(src)> blocks{src, smem_raw, bars, bytes, sb, stages, count};
  const int warp = threadIdx.x >> 5;
  if (warp == N8) {
    if (!blocks.copy(wlim)) {
      if ((threadIdx.x & 31) == 0) atomicOr(status + b, VB_STATUS_WATCHDOG);
      return;
    }
    __syncthreads();   // of the reduction below
    return;
  }
  const int row = sweep_row();
  const bool own = row < n && (threadIdx.x & 3) == 0;
  const double* rin = first ? w.rmod : mv.tmp;
  // operands of a step, three sets in rotation: the right-hand side and the
  // coupling of the layer the step forms an operand for, that layer's row scale
  // (1 for FP64 inverses) and, backward, x of the step's layer
  struct Ops {
    double vec, cpl, sc, x;
  };
  int loaded = 0;
  auto load = [&](Ops& o) {
    const int s = loaded++;
    o.vec = o.cpl = o.x = 0.0;
    o.sc = 1.0;
    if (!own || s >= count) return;
    if (s < F) {
      const int64_t at = (int64_t)s * n + row;   // forms r'_{s+1}
      o.vec = rin[at + n];
      o.cpl = w.subn[at];
      if (!f64) o.sc = mv.rs[at + n];
    } else {
      const int64_t at = (int64_t)(count - 1 - s) * n + row;   // c of this layer, the operand of the one below
      if (!first) o.x = xb[at];
      if (s < count - 1) {
        o.vec = mv.tmp[at - n];
        o.cpl = w.supn[at - n];
        if (!f64) o.sc = mv.rs[at - n];
      }
    }
  };
  double cmax = 0.0, xmax = 0.0;
  bool bad = false;
  // r'_{nz-2}, formed in the step that starts by loading the operands of the
  // first backward step (which needs it); the later ones read this thread's
  // earlier stores
  double turn = 0.0;
  auto step = [&](int s, const Ops& c, Ops& f) {
    load(f);
    const double* vc = v + (s & 1) * VB_MAX_NI;
    double* vn = v + ((s + 1) & 1) * VB_MAX_NI;
    const double u = f64 ? row_dot<N8>(reinterpret_cast<const double*>(blocks.block()), n, ld, row, vc)
                         : row_dot<N8>(reinterpret_cast<const float*>(blocks.block()), n, ldf, row, vc);
    if (own) {
      const double x = (s == F && F >= 2 ? turn : c.vec) - c.cpl * u;
      vn[row] = c.sc * x;
      if (s == F - 2) turn = x;
      if (s < F) {
        mv.tmp[(int64_t)(s + 1) * n + row] = x;
      } else {
        const double xn = first ? u : c.x + u;
        xb[(int64_t)(count - 1 - s) * n + row] = xn;
        cmax = fmax(cmax, fabs(u));
        xmax = fmax(xmax, fabs(xn));
        bad |= !isfinite(xn);
      }
    }
    blocks.next();
    blocks.used();
    return __syncthreads_or(0) == 0;
  };
  if (own) {
    const double r0 = rin[row];
    v[row] = (f64 ? 1.0 : mv.rs[row]) * r0;
    mv.tmp[row] = r0;
  }
  Ops o0, o1, o2;
  load(o0);
  load(o1);
  if (__syncthreads_or(0)) return;   // v written, the first block there
  for (int s = 0; s < count; s += 3) {
    if (!step(s, o0, o2)) return;
    if (s + 1 >= count) break;
    if (!step(s + 1, o1, o0)) return;
    if (s + 2 >= count) break;
    if (!step(s + 2, o2, o1)) return;
  }
  // ---- convergence of this atmosphere
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    cmax = fmax(cmax, __shfl_xor_sync(0xffffffffu, cmax, off));
    xmax = fmax(xmax, __shfl_xor_sync(0xffffffffu, xmax, off));
  }
  const int anybad = __any_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    red[warp][0] = cmax;
    red[warp][1] = xmax;
    redb[warp] = anybad;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double cm2 = red[0][0], xm2 = red[0][1];
    int nb = redb[0];
    for (int q = 1; q < N8; ++q) {
      cm2 = fmax(cm2, red[q][0]);
      xm2 = fmax(xm2, red[q][1]);
      nb |= redb[q];
    }
    if (passes) passes[b] += 1;
    if (first) {
      if (md != MX_FP64) mode[b] = MX_REFINE;
    } else if (!nb && cm2 <= tol * xm2) {
      mode[b] = MX_DONE;
    }
  }
}

// Mode bookkeeping between the passes (one thread per atmosphere):
//  op 0 (after the FP32 factor): an FP32 zero pivot, non-finite inverse or
//        watchdog sends the atmosphere to MX_FP64 (todo = 1); status32 is
//        cleared.
//  op 1 (after the refinement passes): MX_REFINE atmospheres stalled: to
//        MX_FP64 with VB_STATUS_REFINE_STALL (todo = 1); others todo = 0.
__global__ void mx_mode_kernel(int batch, int op, int32_t* __restrict__ mode, int32_t* __restrict__ todo,
                               int32_t* __restrict__ status32, int32_t* __restrict__ status) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  int t = 0;
  if (op == 0) {
    const bool failed = (status32[b] & (VB_STATUS_ZERO_PIVOT | VB_STATUS_NONFINITE | VB_STATUS_WATCHDOG)) != 0;
    mode[b] = failed ? MX_FP64 : MX_REFINE;
    if (status32[b] & VB_STATUS_WATCHDOG) status[b] |= VB_STATUS_WATCHDOG;
    status32[b] = 0;
    t = failed;
  } else if (mode[b] == MX_REFINE) {
    mode[b] = MX_FP64;
    status[b] |= VB_STATUS_REFINE_STALL;
    t = 1;
  }
  todo[b] = t;
}

// sol = y + 3/(2r) k1 + 1/(2r) k2, delta = |sol - (y + k1/r)| (jax_step.py:313-314)
// from the refined stage vectors (k1 rows, k2 in the aux rows).
__global__ void mx_finish_kernel(Batch B, const double* __restrict__ ws, const double* __restrict__ y,
                                 double* __restrict__ sol, double* __restrict__ delta, int32_t* __restrict__ status) {
  const int b = blockIdx.y, j = blockIdx.x;
  const Geo g = geo_of(B, b);
  if (j >= g.nz) return;
  const int n = B.ni;
  WsView w = ws_view(const_cast<double*>(ws), g, n, B.ld);
  const double r = ros2_r();
  bool bad = false;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int64_t e = g.z0 * n + (int64_t)j * n + i;
    const double k1 = w.k1[(int64_t)j * n + i], k2 = w.aux[(int64_t)j * n + i], yv = y[e];
    const double s = yv + (3.0 / (2.0 * r)) * k1 + (1.0 / (2.0 * r)) * k2;
    const double yk2 = yv + k1 / r;
    sol[e] = s;
    delta[e] = fabs(s - yk2);
    bad |= !isfinite(s);
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(status + b, VB_STATUS_NONFINITE);
}

template <int N8>
static cudaError_t launch_mx_pass_t(const Batch& B, double* ws, void* mxr, int xsel, bool first, int32_t* mode,
                                    const int32_t* only, int32_t* passes, double tol, int32_t* status,
                                    long long wlim, cudaStream_t st) {
  if (!first) {
    dim3 grid(B.nz, B.count);
    mx_residual_kernel<N8><<<grid, 32 * N8, 0, st>>>(B, ws, mxr, xsel, mode, only);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  // as deep a ring as fits, or as lets two CTAs share an SM
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int stages = SWEEP_MAX_STAGES;
  while (B.count > sms && stages > 2 && 2 * mx_pass_smem(B.ni, stages) > 224 * 1024) --stages;
  while (stages > 1 && mx_pass_smem(B.ni, stages) > 220 * 1024) --stages;
  const size_t sm = mx_pass_smem(B.ni, stages);
  cudaError_t e = cudaFuncSetAttribute(mx_sweep_kernel<N8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  mx_sweep_kernel<N8><<<B.count, 32 * N8 + 32, sm, st>>>(B, ws, mxr, xsel, first, mode, only, passes, tol, status,
                                                         stages, wlim);
  return cudaGetLastError();
}

template <int N8 = 1>
static cudaError_t launch_mx_pass_n(int n8, const Batch& B, double* ws, void* mxr, int xsel, bool first,
                                    int32_t* mode, const int32_t* only, int32_t* passes, double tol, int32_t* status,
                                    long long wlim, cudaStream_t st) {
  if constexpr (N8 < VB_MAX_NI / 8)
    if (n8 > N8) return launch_mx_pass_n<N8 + 1>(n8, B, ws, mxr, xsel, first, mode, only, passes, tol, status, wlim, st);
  return launch_mx_pass_t<N8>(B, ws, mxr, xsel, first, mode, only, passes, tol, status, wlim, st);
}

cudaError_t launch_mx_pass(const Batch& B, double* ws, void* mxr, int xsel, bool first, int32_t* mode,
                           const int32_t* only, int32_t* passes, double tol, int32_t* status, cudaStream_t st) {
  return launch_mx_pass_n((B.ni + 7) / 8, B, ws, mxr, xsel, first, mode, only, passes, tol, status, wait_limit(), st);
}

cudaError_t launch_mx_mode(int batch, int op, int32_t* mode, int32_t* todo, int32_t* status32, int32_t* status,
                           cudaStream_t st) {
  mx_mode_kernel<<<(batch + 127) / 128, 128, 0, st>>>(batch, op, mode, todo, status32, status);
  return cudaGetLastError();
}

cudaError_t launch_mx_finish(const Batch& B, const double* ws, const double* y, double* sol, double* delta,
                             int32_t* status, cudaStream_t st) {
  dim3 grid(B.nz, B.count);
  mx_finish_kernel<<<grid, 128, 0, st>>>(B, ws, y, sol, delta, status);
  return cudaGetLastError();
}

}  // namespace vb
