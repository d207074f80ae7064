// FEM operators, persistent CG solvers and the FEM/BEM demag pipeline on the device.
//
// Pipeline per call (DemagFieldLindholmGPU.compute_vec, gpu/fields/Demag_Lindholm_GPU.py:643-670):
//   b  = Ms int grad v . m                      k_div   (difference form)
//   u1 : A u1 = b - mean(b), u1 -= mean(u1)     k_cg / k_cg_ir  (:569-582; PETSc CG+GAMG there)
//   g  = B u1|bnd                               dense GEMV or H-matrix (:585-616)
//   u2 : A_II u_I = -A_IB g, u2|bnd = g          k_u2rhs + k_cg / k_cg_ir  (:618-640)
//   phi = u1 + u2 ;  H = G phi / V_i            k_grad  (:659-670)
// The Dirichlet problem is solved on the interior unknowns only; DOLFINx's identity rows for
// the boundary dofs (assemble_matrix with bcs) give the same interior solution.  CG stops when
// ||r||_2 <= max(rtol ||b||_2, atol) (unpreconditioned residual, the KSP default test with a
// zero initial guess) or after maxit.
//
// Persistent solvers: one cooperative launch per solve, one CTA of 1024 threads per SM.  Each
// reduction writes one partial per CTA; after the grid barrier every CTA sums the partials in
// the same order (deterministic, no contended atomics).  Every barrier wait is bounded.
#include <algorithm>
#include <cmath>

#include "fem.cuh"

namespace spx {

// ------------------------------------------------------------------ SELL kernels
// one warp per 32-row slice; thread = row
#define SELL_ROW_LOOP(nslices, ...)                                                    \
  {                                                                                     \
    const int lane_ = threadIdx.x & 31;                                                 \
    const int64_t gw_ = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;           \
    const int64_t nw_ = (gridDim.x * (int64_t)blockDim.x) >> 5;                          \
    for (int64_t sl_ = gw_; sl_ < (nslices); sl_ += nw_) {                              \
      const int64_t row = sl_ * 32 + lane_;                                             \
      const int64_t base_ = sp[sl_];                                                    \
      const int width = static_cast<int>((sp[sl_ + 1] - base_) >> 5);                   \
      __VA_ARGS__                                                                       \
    }                                                                                   \
  }

// b_i = sum_j D_ij . (m_j - m_i) + Dsum_i . m_i
template <class TV, class TM>
__global__ void k_div(int64_t n, int64_t nslices, const int64_t* __restrict__ sp, const int32_t* __restrict__ col,
                      const TM* __restrict__ D, int64_t L, const double* __restrict__ Dsum, const TV* __restrict__ m,
                      TV* __restrict__ b) {
  SELL_ROW_LOOP(nslices, {
    if (row < n) {
      const TV mx = m[3 * row], my = m[3 * row + 1], mz = m[3 * row + 2];
      TV acc = 0;
      for (int k = 0; k < width; ++k) {
        const int64_t idx = base_ + ((int64_t)k << 5) + lane_;
        const int64_t j = col[idx];
        acc += static_cast<TV>(D[idx]) * (m[3 * j] - mx) + static_cast<TV>(D[L + idx]) * (m[3 * j + 1] - my) +
               static_cast<TV>(D[2 * L + idx]) * (m[3 * j + 2] - mz);
      }
      acc += static_cast<TV>(Dsum[row]) * mx + static_cast<TV>(Dsum[n + row]) * my +
             static_cast<TV>(Dsum[2 * n + row]) * mz;
      b[row] = acc;
    }
  })
}

// H_i = sum_j Gv_ij (phi_j - phi_i)
template <class TV, class TM>
__global__ void k_grad(int64_t n, int64_t nslices, const int64_t* __restrict__ sp, const int32_t* __restrict__ col,
                       const TM* __restrict__ Gv, int64_t L, const TV* __restrict__ phi, TV* __restrict__ H) {
  SELL_ROW_LOOP(nslices, {
    if (row < n) {
      const TV pi = phi[row];
      TV hx = 0, hy = 0, hz = 0;
      for (int k = 0; k < width; ++k) {
        const int64_t idx = base_ + ((int64_t)k << 5) + lane_;
        const TV p = phi[col[idx]] - pi;
        hx += static_cast<TV>(Gv[idx]) * p;
        hy += static_cast<TV>(Gv[L + idx]) * p;
        hz += static_cast<TV>(Gv[2 * L + idx]) * p;
      }
      H[3 * row] = hx;
      H[3 * row + 1] = hy;
      H[3 * row + 2] = hz;
    }
  })
}

template <class TV>
__global__ void k_u2rhs(int64_t n, int64_t nslices, const int64_t* __restrict__ sp, const int32_t* __restrict__ col,
                        const double* __restrict__ v, const TV* __restrict__ g, TV* __restrict__ b) {
  SELL_ROW_LOOP(nslices, {
    if (row < n) {
      double acc = 0;
      for (int k = 0; k < width; ++k) {
        const int64_t idx = base_ + ((int64_t)k << 5) + lane_;
        acc += v[idx] * static_cast<double>(g[col[idx]]);
      }
      b[row] = static_cast<TV>(-acc);
    }
  })
}

template <class TV>
__global__ void k_phi_interior(int64_t NI, const int32_t* __restrict__ interior, const TV* __restrict__ u1,
                               const TV* __restrict__ xI, TV* __restrict__ phi) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < NI) {
    const int32_t g = interior[i];
    phi[g] = u1[g] + xI[i];
  }
}

template <class T>
__global__ void k_gather_idx(int64_t n, const int32_t* __restrict__ idx, const T* __restrict__ src, T* __restrict__ dst) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[idx[i]];
}

// dense B (FP64, row-major Nb x Nb): warp per row; g = B xb ; phi[bverts] = u1 + g
template <class TV>
__global__ void k_dense_gemv(int64_t Nb, const double* __restrict__ B, const TV* __restrict__ xb,
                             const int32_t* __restrict__ bverts, const TV* __restrict__ u1, TV* __restrict__ phi,
                             TV* __restrict__ gB) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (gridDim.x * (int64_t)blockDim.x) >> 5;
  for (int64_t i = w; i < Nb; i += nw) {
    const double* row = B + i * Nb;
    double acc = 0.0;
    for (int64_t j = lane; j < Nb; j += 32) acc += row[j] * static_cast<double>(xb[j]);
    acc = warp_sum(acc);
    if (lane == 0) {
      const TV y = static_cast<TV>(acc);
      gB[i] = y;
      if (phi) phi[bverts[i]] = u1[bverts[i]] + y;
    }
  }
}

// Component means of ensembles (node offsets `off`), in two passes over chunks of SEG_CH
// entries so that every component, however large, is spread over many CTAs: k_seg_sum writes
// the chunk sums part[seg][c]; the apply kernels sum a component's chunk sums in a fixed order
// (the same mean in every CTA, deterministic) and remove the mean from their chunk.
constexpr int SEG_CH = 8192;

// chunk sums of x, or of y sdinv when y is given: the FP64 state (of y without sdinv)
template <class TV>
__global__ void k_seg_sum(const int64_t* __restrict__ off, int maxch, const TV* __restrict__ x,
                          const double* __restrict__ y, const double* __restrict__ sdinv, double* __restrict__ part) {
  __shared__ double sh[32];
  const int seg = blockIdx.y, c = blockIdx.x;
  const int64_t a = off[seg] + static_cast<int64_t>(c) * SEG_CH, end = off[seg + 1];
  if (a >= end) return;  // uniform per CTA
  const int64_t e = min(end, a + SEG_CH);
  double v = 0.0;
  for (int64_t i = a + threadIdx.x; i < e; i += blockDim.x) v += y ? (sdinv ? y[i] * sdinv[i] : y[i]) : static_cast<double>(x[i]);
  v = block_sum(v, sh);
  if (threadIdx.x == 0) part[static_cast<int64_t>(seg) * maxch + c] = v;
}

__device__ __forceinline__ double seg_mean(const int64_t* __restrict__ off, int maxch, const double* __restrict__ part,
                                           int seg) {
  const int64_t len = off[seg + 1] - off[seg];
  const int nch = static_cast<int>((len + SEG_CH - 1) / SEG_CH);
  double s = 0.0;
  for (int c = 0; c < nch; ++c) s += part[static_cast<int64_t>(seg) * maxch + c];
  return s / static_cast<double>(len);
}

// remove each component's mean from a projected solution (x = y sdinv when the FP64 state y
// is kept, x = y when it is kept unscaled: no sdinv)
template <class TV>
__global__ void k_seg_center(const int64_t* __restrict__ off, int maxch, const double* __restrict__ part,
                             TV* __restrict__ x, double* __restrict__ y, const double* __restrict__ sdinv) {
  const int seg = blockIdx.y;
  const int64_t a = off[seg] + static_cast<int64_t>(blockIdx.x) * SEG_CH, end = off[seg + 1];
  if (a >= end) return;
  const int64_t e = min(end, a + SEG_CH);
  const double mean = seg_mean(off, maxch, part, seg);
  for (int64_t i = a + threadIdx.x; i < e; i += blockDim.x) {
    if (y) {
      const double sd = sdinv ? sdinv[i] : 1.0;
      const double xv = y[i] * sd - mean;
      x[i] = static_cast<TV>(xv);
      y[i] = xv / sd;
    } else {
      x[i] = static_cast<TV>(static_cast<double>(x[i]) - mean);
    }
  }
}

// bh = (b minus its mean over each component) * sdinv (1 without sdinv), in FP64
template <class TV>
__global__ void k_seg_center_bh(const int64_t* __restrict__ off, int maxch, const double* __restrict__ part,
                                const TV* __restrict__ b, const double* __restrict__ sdinv, double* __restrict__ bh) {
  const int seg = blockIdx.y;
  const int64_t a = off[seg] + static_cast<int64_t>(blockIdx.x) * SEG_CH, end = off[seg + 1];
  if (a >= end) return;
  const int64_t e = min(end, a + SEG_CH);
  const double mean = seg_mean(off, maxch, part, seg);
  for (int64_t i = a + threadIdx.x; i < e; i += blockDim.x) 
    bh[i] = (static_cast<double>(b[i]) - mean) * (sdinv ? sdinv[i] : 1.0);
}

// out = b minus its mean over each component
template <class TV>
__global__ void k_seg_center_b(const int64_t* __restrict__ off, int maxch, const double* __restrict__ part,
                               const TV* __restrict__ b, TV* __restrict__ out) {
  const int seg = blockIdx.y;
  const int64_t a = off[seg] + static_cast<int64_t>(blockIdx.x) * SEG_CH, end = off[seg + 1];
  if (a >= end) return;
  const int64_t e = min(end, a + SEG_CH);
  const double mean = seg_mean(off, maxch, part, seg);
  for (int64_t i = a + threadIdx.x; i < e; i += blockDim.x) out[i] = static_cast<TV>(static_cast<double>(b[i]) - mean);
}

// starting guess: polynomial extrapolation of the stored solutions (order cnt - 1)
__global__ void k_axpy_sub(int64_t n, const double* __restrict__ a, const double* __restrict__ b,
                           double* __restrict__ out, int mode) {  // mode 0: out = a - b; 1: out += a
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = mode == 0 ? a[i] - b[i] : out[i] + a[i];
}

// the stored solutions of a slot, newest first, and the extrapolation weights
// (-1)^k C(cnt, k + 1): the polynomial through the last cnt solutions at the next step
struct ExtrapArgs {
  const double* h[CG_HIST];
  double w[CG_HIST];
  int cnt;
};

template <class T>
__global__ void k_extrap(int64_t n, ExtrapArgs a, T* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double v = 0.0;
#pragma unroll
  for (int k = 0; k < CG_HIST; ++k)
    if (k < a.cnt) v += a.w[k] * a.h[k][i];
  out[i] = static_cast<T>(v);
}

constexpr int CG_BLOCK = 1024;

#define CG_ROWS_BEGIN                                               \
  for (int64_t sl = gw; sl < P.nslices; sl += nw) {                 \
    const int64_t row = sl * 32 + lane;                             \
    const int64_t base = P.sp[sl];                                  \
    const int width = static_cast<int>((P.sp[sl + 1] - base) >> 5); \
    (void)base; (void)width;                                        \
    if (row < n) {
#define CG_ROWS_END \
  }                 \
  }

// ------------------------------------------------------------------ pipelined FP64 CG
struct CgParams {
  int64_t n, nslices;
  const int64_t* sp;
  const int32_t* col;
  const double* val;
  const double* sdinv;
  const double* diag;
  const double* b;
  double* x;
  double *r, *w0, *w1, *p, *s, *z, *y;
  double* part;
  unsigned int* bar;
  int* err;
  int* iters;
  double* resid;
  unsigned long long* iters_acc;
  double* res_acc;
  double rtol, atol;
  int maxit, warm, project;
};

__device__ __forceinline__ double spmv64(const CgParams& P, int64_t base, int width, int lane, const double* v) {
  double acc = 0;
  for (int k = 0; k < width; ++k) {
    const int64_t idx = base + ((int64_t)k << 5) + lane;
    acc += P.val[idx] * v[P.col[idx]];
  }
  return acc;
}

__global__ void __launch_bounds__(CG_BLOCK, 1) k_cg(CgParams P) {
  __shared__ double sh[160];
  const unsigned nb = gridDim.x;
  const int lane = threadIdx.x & 31;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (gridDim.x * (int64_t)blockDim.x) >> 5;
  unsigned int* cnt = P.bar;
  unsigned int* gen = P.bar + 1;
  const int64_t n = P.n;
  double tot[4];
  double meanb = 0.0;
  if (P.project) {
    double part = 0.0;
    CG_ROWS_BEGIN part += P.b[row];
    CG_ROWS_END
    cta_partial(P.part, 0, part, 0.0, 0.0, 0.0, sh);
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
    cta_total(P.part, 0, tot, sh);
    meanb = tot[0] / static_cast<double>(n);
  }
  {
    double bb = 0.0;
    CG_ROWS_BEGIN
      const double bv = P.b[row] - meanb;
      P.r[row] = bv * P.sdinv[row];
      P.y[row] = P.warm ? P.x[row] / P.sdinv[row] : 0.0;
      bb += bv * bv;
    CG_ROWS_END
    cta_partial(P.part, 1, bb, 0.0, 0.0, 0.0, sh);
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
  }
  cta_total(P.part, 1, tot, sh);
  const double bb = tot[0];
  // b = 0: the solution is 0 (a warm start would only iterate on rounding noise)
  const bool warm = P.warm && bb > 0.0;
  if (P.warm && !warm) {
    CG_ROWS_BEGIN P.y[row] = 0.0;
    CG_ROWS_END
  }
  if (warm) {
    CG_ROWS_BEGIN P.r[row] -= spmv64(P, base, width, lane, P.y);
    CG_ROWS_END
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
  }
  {
    double g = 0.0, dl = 0.0, rh = 0.0;
    CG_ROWS_BEGIN
      const double w = spmv64(P, base, width, lane, P.r);
      P.w0[row] = w;
      const double rv = P.r[row];
      g += rv * rv;
      dl += w * rv;
      rh += P.diag[row] * rv * rv;
    CG_ROWS_END
    cta_partial(P.part, 2, g, dl, rh, 0.0, sh);
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
  }
  const double tol2 = fmax(P.rtol * P.rtol * bb, P.atol * P.atol);
  double gprev = 1.0, aprev = 1.0, rho = 0.0, rho0 = -1.0;
  int it = 0;
  for (;; ++it) {
    cta_total(P.part, 2 + (it & 1), tot, sh);
    const double gm = tot[0], dl = tot[1];
    rho = tot[2];
    if (rho0 < 0.0) rho0 = rho;
    if (rho <= tol2 || it >= P.maxit || !(gm > 0.0)) break;
    double beta, alpha;
    if (it == 0) {
      beta = 0.0;
      alpha = gm / dl;
    } else {
      beta = gm / gprev;
      alpha = gm / (dl - beta * gm / aprev);
    }
    const double* wc = (it & 1) ? P.w1 : P.w0;
    double* wn = (it & 1) ? P.w0 : P.w1;
    double g2 = 0.0, d2 = 0.0, r2 = 0.0;
    CG_ROWS_BEGIN
      const double nv = spmv64(P, base, width, lane, wc);
      const double wv = wc[row];
      const double rv = P.r[row];
      double zv, sv, pv;
      if (it == 0) {
        zv = nv; sv = wv; pv = rv;
      } else {
        zv = nv + beta * P.z[row];
        sv = wv + beta * P.s[row];
        pv = rv + beta * P.p[row];
      }
      P.z[row] = zv;
      P.s[row] = sv;
      P.p[row] = pv;
      P.y[row] += alpha * pv;
      const double rn = rv - alpha * sv;
      const double wnv = wv - alpha * zv;
      P.r[row] = rn;
      wn[row] = wnv;
      g2 += rn * rn;
      d2 += wnv * rn;
      r2 += P.diag[row] * rn * rn;
    CG_ROWS_END
    // slot 2 + ((it + 1) & 1) was last read at the top of iteration it - 1, a barrier ago
    cta_partial(P.part, 2 + ((it + 1) & 1), g2, d2, r2, 0.0, sh);
    gprev = gm;
    aprev = alpha;
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
  }
  double sx = 0.0;
  CG_ROWS_BEGIN
    const double xv = P.y[row] * P.sdinv[row];
    P.x[row] = xv;
    sx += xv;
  CG_ROWS_END
  if (P.project) {
    cta_partial(P.part, 0, sx, 0.0, 0.0, 0.0, sh);
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
    cta_total(P.part, 0, tot, sh);
    const double mx = tot[0] / static_cast<double>(n);
    CG_ROWS_BEGIN P.x[row] -= mx;
    CG_ROWS_END
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *P.iters = it;
    *P.resid = bb > 0.0 ? sqrt(rho / bb) : 0.0;
    atomicAdd(P.iters_acc, (unsigned long long)it);
    atomicAdd(P.iters_acc + 1, 1ull);
    atomicAdd(P.iters_acc + 2, 1ull);
    if (bb > 0.0) {
      atomicAdd(P.res_acc, sqrt(fmax(rho0, 0.0) / bb));
      atomicAdd(P.res_acc + 1, sqrt(rho / bb));
    }
  }
}

// ------------------------------------------------------------------ FP32 CG inside FP64 refinement
template <class TV>
struct CgIrParams {
  int64_t n, nslices;
  const int64_t* sp;
  const int32_t* col;
  const float* v32;
  const double* v64;
  const double* sdinv;
  const double* diag;
  const TV* b;
  TV* x;
  double *bh, *y;
  float *r, *p, *q, *s, *d;
  double* part;
  unsigned int* bar;
  int* err;
  int* iters;
  double* resid;
  unsigned long long* iters_acc;
  double* res_acc;  // [0] sum of initial relative residuals, [1] sum of final ones
  double rtol, atol, inner_rtol;
  int maxit, max_outer, inner_maxit, warm, project;
  int bh_given;  // bh already holds the scaled, projected right-hand side (FP64)
};

template <class TV>
__global__ void __launch_bounds__(CG_BLOCK, 1) k_cg_ir(CgIrParams<TV> P) {
  __shared__ double sh[160];
  const unsigned nb = gridDim.x;
  const int lane = threadIdx.x & 31;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (gridDim.x * (int64_t)blockDim.x) >> 5;
  unsigned int* cnt = P.bar;
  unsigned int* gen = P.bar + 1;
  const int64_t n = P.n;
  double tot[4];
  double meanb = 0.0;
  if (P.project && !P.bh_given) {
    double part = 0.0;
    CG_ROWS_BEGIN part += static_cast<double>(P.b[row]);
    CG_ROWS_END
    cta_partial(P.part, 0, part, 0.0, 0.0, 0.0, sh);
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
    cta_total(P.part, 0, tot, sh);
    meanb = tot[0] / static_cast<double>(n);
  }
  {
    double bb = 0.0;
    CG_ROWS_BEGIN
      double bv;
      if (P.bh_given) {
        bv = P.bh[row] / P.sdinv[row];
      } else {
        bv = static_cast<double>(P.b[row]) - meanb;
        P.bh[row] = bv * P.sdinv[row];
      }
      if (!P.warm) P.y[row] = 0.0;
      bb += bv * bv;
    CG_ROWS_END
    cta_partial(P.part, 1, bb, 0.0, 0.0, 0.0, sh);
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
  }
  cta_total(P.part, 1, tot, sh);
  const double bb = tot[0];
  if (P.warm && !(bb > 0.0)) {  // b = 0: the solution is 0
    CG_ROWS_BEGIN P.y[row] = 0.0;
    CG_ROWS_END
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
  }
  const double tol2 = fmax(P.rtol * P.rtol * bb, P.atol * P.atol);
  int total = 0, outers = 0;
  double rho = 0.0, rho0 = -1.0;
  for (int outer = 0; outer < P.max_outer; ++outer) {
    ++outers;
    // true residual in FP64; inner start r = r64 (FP32), d = 0
    {
      double rh = 0.0;
      CG_ROWS_BEGIN
        double acc = 0.0;
        for (int k = 0; k < width; ++k) {
          const int64_t idx = base + ((int64_t)k << 5) + lane;
          acc += P.v64[idx] * P.y[P.col[idx]];
        }
        const double r64 = P.bh[row] - acc;
        rh += P.diag[row] * r64 * r64;
        P.r[row] = static_cast<float>(r64);
        P.d[row] = 0.0f;
      CG_ROWS_END
      cta_partial(P.part, 0, rh, 0.0, 0.0, 0.0, sh);
      if (!grid_barrier(cnt, gen, nb, P.err)) return;
    }
    cta_total(P.part, 0, tot, sh);
    rho = tot[0];
    if (rho0 < 0.0) rho0 = rho;
    if (rho <= tol2 || total >= P.maxit) break;
    // reduce the residual only as far as the target needs (with a 0.3 margin), at most
    // by inner_rtol per refinement step (the FP32 inner solve's reliable range)
    const double need = 0.3 * sqrt(tol2 / rho);
    const double itol = fmax(P.inner_rtol, fmin(need, 0.5));
    // s = A r, slot 2 <- (r,r), (r,s)
    {
      double g = 0.0, dl = 0.0;
      CG_ROWS_BEGIN
        float acc = 0.0f;
        for (int k = 0; k < width; ++k) {
          const int64_t idx = base + ((int64_t)k << 5) + lane;
          acc += P.v32[idx] * P.r[P.col[idx]];
        }
        P.s[row] = acc;
        const double rv = P.r[row];
        g += rv * rv;
        dl += rv * static_cast<double>(acc);
      CG_ROWS_END
      cta_partial(P.part, 2, g, dl, 0.0, 0.0, sh);
      if (!grid_barrier(cnt, gen, nb, P.err)) return;
    }
    double g0 = 0.0, gprev = 1.0, aprev = 1.0;
    for (int it = 0;; ++it) {
      cta_total(P.part, 2 + (it & 1), tot, sh);
      const double gm = tot[0], dl = tot[1];
      if (it == 0) g0 = gm;
      if (gm <= itol * itol * g0 || it >= P.inner_maxit || total >= P.maxit || !(gm > 0.0) ||
          !(dl > 0.0))
        break;
      double beta, alpha;
      if (it == 0) {
        beta = 0.0;
        alpha = gm / dl;
      } else {
        beta = gm / gprev;
        alpha = gm / (dl - beta * gm / aprev);
      }
      const float a = static_cast<float>(alpha), bt = static_cast<float>(beta);
      CG_ROWS_BEGIN
        const float rv = P.r[row], sv = P.s[row];
        const float pv = (it == 0) ? rv : rv + bt * P.p[row];
        const float qv = (it == 0) ? sv : sv + bt * P.q[row];
        P.p[row] = pv;
        P.q[row] = qv;
        P.d[row] += a * pv;
        P.r[row] = rv - a * qv;
      CG_ROWS_END
      if (!grid_barrier(cnt, gen, nb, P.err)) return;
      double g2 = 0.0, d2 = 0.0;
      CG_ROWS_BEGIN
        float acc = 0.0f;
        for (int k = 0; k < width; ++k) {
          const int64_t idx = base + ((int64_t)k << 5) + lane;
          acc += P.v32[idx] * P.r[P.col[idx]];
        }
        P.s[row] = acc;
        const double rv = P.r[row];
        g2 += rv * rv;
        d2 += rv * static_cast<double>(acc);
      CG_ROWS_END
      // slot 2 + ((it+1)&1) was last read at the top of iteration it-1, two barriers ago
      cta_partial(P.part, 2 + ((it + 1) & 1), g2, d2, 0.0, 0.0, sh);
      gprev = gm;
      aprev = alpha;
      ++total;
      if (!grid_barrier(cnt, gen, nb, P.err)) return;
    }
    CG_ROWS_BEGIN P.y[row] += static_cast<double>(P.d[row]);
    CG_ROWS_END
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
  }
  double mx = 0.0;
  if (P.project) {
    double sx = 0.0;
    CG_ROWS_BEGIN sx += P.y[row] * P.sdinv[row];
    CG_ROWS_END
    cta_partial(P.part, 1, sx, 0.0, 0.0, 0.0, sh);
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
    cta_total(P.part, 1, tot, sh);
    mx = tot[0] / static_cast<double>(n);
  }
  CG_ROWS_BEGIN
    const double xv = P.y[row] * P.sdinv[row] - mx;
    P.x[row] = static_cast<TV>(xv);
    P.y[row] = xv / P.sdinv[row];
  CG_ROWS_END
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *P.iters = total;
    *P.resid = bb > 0.0 ? sqrt(rho / bb) : 0.0;
    atomicAdd(P.iters_acc, (unsigned long long)total);
    atomicAdd(P.iters_acc + 1, (unsigned long long)outers);
    atomicAdd(P.iters_acc + 2, 1ull);
    if (bb > 0.0) {
      atomicAdd(P.res_acc, sqrt(fmax(rho0, 0.0) / bb));
      atomicAdd(P.res_acc + 1, sqrt(rho / bb));
    }
  }
}

// number of identical diagonal blocks of the FEM system when every sample of an ensemble has
// the same matrix bit for bit (equal node counts, tets and stiffness values; columns shifted by
// the sample's offset): 2, 4 or 8 such blocks, else 1
int repeated_blocks(const HostFem& fem, const std::vector<int64_t>& off) {
  const int64_t ns = static_cast<int64_t>(off.size()) - 1;
  if (ns != 2 && ns != 4 && ns != 8) return 1;
  const int64_t n1 = off[1] - off[0];
  if (off[0] != 0 || n1 <= AmgOptions{}.coarse_max) return 1;  // the block must have an AMG hierarchy
  for (int64_t s = 1; s <= ns; ++s)
    if (off[s] != s * n1) return 1;
  const int64_t nnz1 = fem.rowptr[n1];
  for (int64_t s = 1; s < ns; ++s) {
    const int64_t r0 = s * n1, k0 = fem.rowptr[r0];
    if (fem.rowptr[r0 + n1] - k0 != nnz1) return 1;
    for (int64_t i = 0; i <= n1; ++i)
      if (fem.rowptr[r0 + i] - k0 != fem.rowptr[i]) return 1;
    for (int64_t k = 0; k < nnz1; ++k)
      if (fem.col[k0 + k] != fem.col[k] + r0 || fem.A[k0 + k] != fem.A[k]) return 1;
  }
  return static_cast<int>(ns);
}

// the stiffness CSR without its exact zeros off the diagonal (edges whose dihedral angles are
// all right ones, about half of the entries of a mesh of cut cubes): the Poisson solvers read
// their matrices tens of times per solve, and a zero term changes no sum
struct PoissonCsr {
  std::vector<int64_t> rp;
  std::vector<int32_t> ci;
  std::vector<double> a;
};
PoissonCsr drop_zeros(const HostFem& fem) {
  PoissonCsr o;
  o.rp.assign(fem.N + 1, 0);
  o.ci.reserve(fem.col.size());
  o.a.reserve(fem.col.size());
  for (int64_t i = 0; i < fem.N; ++i) {
    for (int64_t k = fem.rowptr[i]; k < fem.rowptr[i + 1]; ++k)
      if (fem.A[k] != 0.0 || fem.col[k] == i) {
        o.ci.push_back(fem.col[k]);
        o.a.push_back(fem.A[k]);
      }
    o.rp[i + 1] = static_cast<int64_t>(o.ci.size());
  }
  return o;
}

// ------------------------------------------------------------------ CgSystem
template <class TM>
void CgSystem<TM>::setup(const HostSell& s, const std::vector<double>& vals_sell, const std::vector<double>& d,
                         int nrep) {
  SPX_CHECK(nrep >= 1, "at least one block");
  reps = nrep;
  n1 = s.nrows;
  n = n1 * reps;
  P.upload(s);
  std::vector<double> v64(vals_sell.size(), 0.0), sd(n1);
  for (int64_t i = 0; i < n1; ++i) {
    SPX_CHECK(d[i] > 0.0, "CG system has a non-positive diagonal");
    sd[i] = 1.0 / std::sqrt(d[i]);
  }
  for (int64_t sl = 0; sl < s.nslices; ++sl) {
    const int64_t w = (s.slice_ptr[sl + 1] - s.slice_ptr[sl]) / SELL_C;
    for (int64_t k = 0; k < w; ++k)
      for (int l = 0; l < SELL_C; ++l) {
        const int64_t idx = s.slice_ptr[sl] + k * SELL_C + l;
        const int64_t row = sl * SELL_C + l;
        v64[idx] = (row < n1) ? vals_sell[idx] * sd[row] * sd[s.col[idx]] : 0.0;
      }
  }
  std::vector<TM> vt(v64.begin(), v64.end());
  vals.upload(vt);
  {  // per-row FP64 data, repeated for every block
    std::vector<double> sdr(n), dr(n);
    for (int r = 0; r < reps; ++r)
      for (int64_t i = 0; i < n1; ++i) {
        sdr[r * n1 + i] = sd[i];
        dr[r * n1 + i] = d[i];
      }
    sdinv64.upload(sdr);
    diag64.upload(dr);
  }
  if (sizeof(TM) == sizeof(float)) {
    vals64.upload(v64);
    y64.alloc(n);
    y64.zero();
    bh64.alloc(n);
    work.alloc(5 * static_cast<size_t>(n) * sizeof(float));
  } else {
    work.alloc(7 * static_cast<size_t>(n) * sizeof(double));
  }
  bar.alloc(2);
  err.alloc(1);
  iters.alloc(1);
  resid.alloc(1);
  iters_acc.alloc(4);
  iters_acc.zero();
  res_acc.alloc(2);
  res_acc.zero();
  int dev;
  SPX_CUDA(cudaGetDevice(&dev));
  int per_sm = 0;
  block = CG_BLOCK;
  if (sizeof(TM) == sizeof(float))
    SPX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cg_ir<double>, CG_BLOCK, 0));
  else
    SPX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cg, CG_BLOCK, 0));
  SPX_CHECK(per_sm > 0, "CG kernel cannot be resident");
  const int64_t want = (s.nslices * 32 + CG_BLOCK - 1) / CG_BLOCK;
  grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(want, num_sms(dev))));
  part.alloc(4 * 4 * static_cast<size_t>(grid));
}

template <class TM>
template <class TV>
CgStats CgSystem<TM>::solve(const TV* b, TV* x, double rtol, double atol, int maxit, bool warm, bool project,
                            int slot, cudaStream_t st, bool sync_stats, int kind) {
  if (kind < 0) kind = slot < 4 ? 0 : (slot < 8 ? 1 : 2);
  if (kind != last_kind) warm = false;
  last_kind = kind;
  const bool use_amg = static_cast<bool>(amg);
  SPX_CHECK(reps == 1 || use_amg, "a system of repeated blocks is solved by the AMG PCG only");
  const bool ir = sizeof(TM) == sizeof(float) || use_amg;  // solution state kept in y64
  SPX_CHECK(ir || sizeof(TV) == sizeof(double), "FP64 CG needs FP64 vectors");
  if (slot >= 0) {
    SPX_CHECK(slot < CG_SLOTS, "extrapolation slot out of range");
    for (int k = 0; k < CG_HIST; ++k)
      if (!hist[slot][k].n) hist[slot][k].alloc(n);
    if (hcount[slot] > 0) {
      ExtrapArgs ea{};
      ea.cnt = hcount[slot];
      double binom = 1.0;  // C(cnt, k + 1), built up term by term
      for (int k = 0; k < CG_HIST; ++k) {
        ea.h[k] = hist[slot][(hhead[slot] + 2 * CG_HIST - 1 - k) % CG_HIST].p;  // newest first
        binom = binom * (ea.cnt - k) / (k + 1);
        ea.w[k] = k < ea.cnt ? ((k % 2) ? -binom : binom) : 0.0;
      }
      double* target = ir ? y64.p : reinterpret_cast<double*>(x);
      k_extrap<double><<<grid_for(n, 256), 256, 0, st>>>(n, ea, target);
      SPX_LAUNCH_CHECK();
      warm = true;
      if (stage_correct) {
        if (slot == 0) {
          if (!pred0.n) pred0.alloc(n);
          SPX_CUDA(cudaMemcpyAsync(pred0.p, target, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
          have_pred0 = true;
        } else if (slot < 4 && have_delta) {
          k_axpy_sub<<<grid_for(n, 256), 256, 0, st>>>(n, delta.p, nullptr, target, 1);
          SPX_LAUNCH_CHECK();
        }
      }
    }
  }
  SPX_CUDA(cudaMemsetAsync(bar.p, 0, bar.bytes(), st));
  SPX_CUDA(cudaMemsetAsync(err.p, 0, err.bytes(), st));
  // ensembles: every component's right-hand side projected on its own (FP64 for the solvers
  // that keep an FP64 state, so that no FP32 rounding leaves a component inconsistent)
  const bool seg = project && seg_off.n > 1;
  const dim3 sgrid(static_cast<unsigned>(std::max(seg_maxch, 1)), static_cast<unsigned>(seg_off.n > 1 ? seg_off.n - 1 : 1));
  if (seg) {
    k_seg_sum<TV><<<sgrid, 256, 0, st>>>(seg_off.p, seg_maxch, b, nullptr, nullptr, seg_part.p);
    SPX_LAUNCH_CHECK();
  }
  const double* seg_sd = use_amg ? nullptr : sdinv64.p;  // the AMG PCG keeps its state unscaled
  if (seg && ir) {
    k_seg_center_bh<TV><<<sgrid, 256, 0, st>>>(seg_off.p, seg_maxch, seg_part.p, b, seg_sd, bh64.p);
    SPX_LAUNCH_CHECK();
  } else if (seg) {
    if (bseg.n < n * sizeof(TV)) bseg.alloc(n * sizeof(TV));
    TV* bc = reinterpret_cast<TV*>(bseg.p);
    k_seg_center_b<TV><<<sgrid, 256, 0, st>>>(seg_off.p, seg_maxch, seg_part.p, b, bc);
    SPX_LAUNCH_CHECK();
    b = bc;
  }
  if (use_amg) {
    launch_amg<TV>(b, x, rtol, atol, maxit, warm, project, st, seg);
  } else if (sizeof(TM) == sizeof(float)) {
    CgIrParams<TV> q;
    q.n = n; q.nslices = P.nslices; q.sp = P.slice_ptr.p; q.col = P.col.p;
    q.v32 = reinterpret_cast<const float*>(vals.p); q.v64 = vals64.p; q.sdinv = sdinv64.p; q.diag = diag64.p;
    q.b = b; q.x = x;
    q.bh = bh64.p; q.y = y64.p;
    float* Wf = reinterpret_cast<float*>(work.p);
    q.r = Wf; q.p = Wf + n; q.q = Wf + 2 * n; q.s = Wf + 3 * n; q.d = Wf + 4 * n;
    q.part = part.p; q.bar = bar.p; q.err = err.p; q.iters = iters.p; q.resid = resid.p;
    q.iters_acc = iters_acc.p;
    q.res_acc = res_acc.p;
    q.rtol = rtol; q.atol = atol; q.inner_rtol = inner_rtol;
    q.maxit = maxit; q.max_outer = max_outer; q.inner_maxit = maxit; q.warm = warm ? 1 : 0;
    q.bh_given = seg ? 1 : 0;
    q.project = project ? 1 : 0;
    void* a2[] = {&q};
    SPX_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(k_cg_ir<TV>), dim3(grid), dim3(block), a2, 0, st));
  } else {
    CgParams p;
    p.n = n; p.nslices = P.nslices; p.sp = P.slice_ptr.p; p.col = P.col.p;
    p.val = reinterpret_cast<const double*>(vals.p); p.sdinv = sdinv64.p; p.diag = diag64.p;
    p.b = reinterpret_cast<const double*>(b); p.x = reinterpret_cast<double*>(x);
    double* W = reinterpret_cast<double*>(work.p);
    p.r = W; p.w0 = W + n; p.w1 = W + 2 * n; p.p = W + 3 * n; p.s = W + 4 * n; p.z = W + 5 * n; p.y = W + 6 * n;
    p.part = part.p; p.bar = bar.p; p.err = err.p; p.iters = iters.p; p.resid = resid.p;
    p.iters_acc = iters_acc.p;
    p.res_acc = res_acc.p;
    p.rtol = rtol; p.atol = atol; p.maxit = maxit; p.warm = warm ? 1 : 0; p.project = project ? 1 : 0;
    void* args[] = {&p};
    SPX_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(k_cg), dim3(grid), dim3(block), args, 0, st));
  }
  if (project && seg_off.n > 1) {
    k_seg_sum<TV><<<sgrid, 256, 0, st>>>(seg_off.p, seg_maxch, x, ir ? y64.p : nullptr, seg_sd, seg_part.p);
    SPX_LAUNCH_CHECK();
    k_seg_center<TV><<<sgrid, 256, 0, st>>>(seg_off.p, seg_maxch, seg_part.p, x, ir ? y64.p : nullptr, seg_sd);
    SPX_LAUNCH_CHECK();
  }
  if (slot == 0 && stage_correct && have_pred0) {  // stage 1's prediction error
    if (!delta.n) delta.alloc(n);
    k_axpy_sub<<<grid_for(n, 256), 256, 0, st>>>(n, ir ? y64.p : reinterpret_cast<const double*>(x), pred0.p,
                                                 delta.p, 0);
    SPX_LAUNCH_CHECK();
    have_delta = true;
    have_pred0 = false;
  }
  if (slot >= 0) {
    double* dst = hist[slot][hhead[slot]].p;
    const double* src = ir ? y64.p : reinterpret_cast<const double*>(x);
    SPX_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
    hhead[slot] = (hhead[slot] + 1) % CG_HIST;
    hcount[slot] = std::min(CG_HIST, hcount[slot] + 1);
  }
  CgStats out;
  if (sync_stats) {
    int h_err = 0, h_it = 0;
    double h_res = 0.0;
    SPX_CUDA(cudaMemcpyAsync(&h_err, err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    SPX_CUDA(cudaMemcpyAsync(&h_it, iters.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    SPX_CUDA(cudaMemcpyAsync(&h_res, resid.p, sizeof(double), cudaMemcpyDeviceToHost, st));
    SPX_CUDA(cudaStreamSynchronize(st));
    if (h_err) throw Error(ERR_TIMEOUT, "CG grid barrier timed out");
    out.iterations = h_it;
    out.rel_residual = h_res;
    out.converged = (h_res <= rtol || h_it < maxit) ? 1 : 0;
  }
  return out;
}

template <class TM>
void CgSystem<TM>::set_segments(const std::vector<int64_t>& offsets, cudaStream_t s) {
  seg_off.upload(offsets, s);
  int64_t mx = 0;
  for (size_t k = 0; k + 1 < offsets.size(); ++k) mx = std::max<int64_t>(mx, offsets[k + 1] - offsets[k]);
  seg_maxch = static_cast<int>((mx + SEG_CH - 1) / SEG_CH);
  const int64_t nseg = offsets.size() > 1 ? static_cast<int64_t>(offsets.size()) - 1 : 1;
  seg_part.alloc(static_cast<size_t>(nseg * std::max(seg_maxch, 1)));
}

template struct CgSystem<double>;
template struct CgSystem<float>;
template CgStats CgSystem<double>::solve<double>(const double*, double*, double, double, int, bool, bool, int,
                                                 cudaStream_t, bool, int);
template CgStats CgSystem<float>::solve<double>(const double*, double*, double, double, int, bool, bool, int,
                                                cudaStream_t, bool, int);
template CgStats CgSystem<float>::solve<float>(const float*, float*, double, double, int, bool, bool, int,
                                               cudaStream_t, bool, int);

// ------------------------------------------------------------------ demag context
template <class TV, class TM>
void DemagCtx<TV, TM>::create(const double* X, int64_t N_, const int32_t* tets, int64_t E_, double Ms_,
                              const DemagOptions& o, cudaStream_t s) {
  SPX_CUDA(cudaGetDevice(&device));
  N = N_;
  E = E_;
  Ms = Ms_;
  opt = o;
  bd.create(X, N, tets, E);
  Nb = bd.host.Nb;
  assemble_fem(X, N, tets, E, fem);
  const int64_t nnz = fem.rowptr[N];
  std::vector<int32_t> all(N);
  for (int64_t i = 0; i < N; ++i) all[i] = static_cast<int32_t>(i);
  build_sell(fem.rowptr, fem.col, all, nullptr, hsell);
  P.upload(hsell, s);
  {
    std::vector<TM> v;
    sell_values<TM>(hsell, fem.Div.data(), 3, true, nnz, Ms, v);
    Div.upload(v, s);
    std::vector<double> ds(3 * N, 0.0);
    for (int64_t i = 0; i < N; ++i)
      for (int64_t k = fem.rowptr[i]; k < fem.rowptr[i + 1]; ++k)
        for (int c = 0; c < 3; ++c) ds[c * N + i] += Ms * fem.Div[3 * k + c];
    Dsum.upload(ds, s);
    std::vector<double> g = fem.G;
    for (int64_t i = 0; i < N; ++i)
      for (int64_t k = fem.rowptr[i]; k < fem.rowptr[i + 1]; ++k)
        for (int c = 0; c < 3; ++c) g[3 * k + c] /= fem.vol[i];
    sell_values<TM>(hsell, g.data(), 3, true, nnz, 1.0, v);
    Gv.upload(v, s);
  }
  vol.upload(fem.vol, s);
  const PoissonCsr K = drop_zeros(fem);
  {
    // an ensemble whose samples all have the same stiffness matrix (a batch of one mesh): the
    // u1 system is that block repeated on the diagonal; its matrix and AMG hierarchy are stored
    // once and the PCG runs on all blocks together (2, 4 or 8 of them)
    const int reps = (opt.backend == 2 && opt.u1_pc == 0) ? repeated_blocks(fem, opt.sample_offsets) : 1;
    const int64_t n1 = N / reps, nnz1 = K.rp[n1];
    const std::vector<int64_t> rp1(K.rp.begin(), K.rp.begin() + n1 + 1);
    const std::vector<int32_t> col1(K.ci.begin(), K.ci.begin() + nnz1);
    const std::vector<double> A1(K.a.begin(), K.a.begin() + nnz1);
    const std::vector<int32_t> rows1(all.begin(), all.begin() + n1);
    HostSell hs1;
    build_sell(rp1, col1, rows1, nullptr, hs1);
    std::vector<double> a1, d1(n1);
    sell_values<double>(hs1, A1.data(), 1, true, nnz1, 1.0, a1);
    for (int64_t i = 0; i < n1; ++i)
      for (int64_t k = rp1[i]; k < rp1[i + 1]; ++k)
        if (col1[k] == i) d1[i] = A1[k];
    cg1.setup(hs1, a1, d1, reps);
    if (opt.u1_pc == 0) cg1.enable_amg(hs1, rp1, col1, A1, d1, true, s);
    SPX_CHECK(reps == 1 || static_cast<bool>(cg1.amg), "no AMG hierarchy for the repeated block");
    cg1.stage_correct = opt.warm_start == 3;
  }
  std::vector<int32_t> bmap(N, -1), imap(N, -1), inter;
  for (int64_t k = 0; k < Nb; ++k) bmap[bd.host.bverts[k]] = static_cast<int32_t>(k);
  for (int64_t i = 0; i < N; ++i)
    if (bmap[i] < 0) {
      imap[i] = static_cast<int32_t>(inter.size());
      inter.push_back(static_cast<int32_t>(i));
    }
  NI = static_cast<int64_t>(inter.size());
  interior.upload(inter, s);
  bverts.upload(bd.host.bverts, s);
  if (NI > 0) {
    HostSell sII, sIB;
    const int64_t nk = K.rp[N];
    build_sell(K.rp, K.ci, inter, &imap, sII);
    build_sell(K.rp, K.ci, inter, &bmap, sIB);
    std::vector<double> aII, aIB;
    sell_values<double>(sII, K.a.data(), 1, true, nk, 1.0, aII);
    sell_values<double>(sIB, K.a.data(), 1, true, nk, 1.0, aIB);
    std::vector<double> d(NI);
    for (int64_t q = 0; q < NI; ++q) {
      const int64_t i = inter[q];
      for (int64_t k = K.rp[i]; k < K.rp[i + 1]; ++k)
        if (K.ci[k] == i) d[q] = K.a[k];
    }
    cg2.setup(sII, aII, d);
    cg2.stage_correct = opt.warm_start == 3;
    PIB.upload(sIB, s);
    AIB.upload(aIB, s);
  }
  if (opt.backend == 0) {
    SPX_CHECK(Nb * Nb * 8 <= (int64_t)64 * 1024 * 1024 * 1024, "dense boundary operator too large");
    Bdense.alloc(static_cast<size_t>(Nb * Nb));
    bd.dense_B(Bdense.p, s);
  } else if (opt.backend == 2) {
    block_boundary_build<TM>(blk, bd, X, N, tets, E, opt, s);
    cg1.set_segments(opt.sample_offsets, s);
  } else {
    if (opt.preset) {
      SPX_CHECK(opt.preset->Nb == Nb && opt.preset->packed, "the given H-matrix does not belong to this boundary");
      H = std::move(*opt.preset);
      opt.preset = nullptr;
      if (H.prec != opt.hprec) H.pack(opt.hprec, s);
    } else {
      H.build(bd, opt.hcfg, s);
      H.pack(opt.hprec, s);
    }
  }
  b.alloc(N); u1.alloc(N); phi.alloc(N); gB.alloc(Nb); xb.alloc(Nb);
  bI.alloc(std::max<int64_t>(NI, 1));
  xI.alloc(std::max<int64_t>(NI, 1));
  u1.zero(s);
  xI.zero(s);
  SPX_CUDA(cudaStreamSynchronize(s));
}

template <class TV, class TM>
void DemagCtx<TV, TM>::potential(const TV* m, cudaStream_t s, bool sync_stats, int slot) {
  const int threads = 256;
  const bool warm = opt.warm_start != 0;
  const int sl = (opt.warm_start >= 2) ? slot : -1;
  const int kind = slot < 4 ? 0 : (slot < 8 ? 1 : 2);  // forward (slot -1 included), adjoint, tangent
  prof.mark(PC_DIV, s);
  k_div<TV, TM><<<grid_for(P.nslices * 32, threads), threads, 0, s>>>(N, P.nslices, P.slice_ptr.p, P.col.p, Div.p,
                                                                     P.len, Dsum.p, m, b.p);
  SPX_LAUNCH_CHECK();
  prof.mark(PC_DIV, s);
  prof.launches[PC_DIV] += 1;
  prof.mark(PC_CG1, s);
  last1 = cg1.template solve<TV>(b.p, u1.p, opt.rtol_u1, opt.atol, opt.maxit_u1, warm, true, sl, s, sync_stats, kind);
  prof.mark(PC_CG1, s);
  prof.launches[PC_CG1] += 1 + (sl >= 0 && cg1.hcount[sl] > 1 ? 1 : 0);
  prof.mark(PC_BND, s);
  if (opt.backend == 0) {
    k_gather_idx<TV><<<grid_for(Nb, 256), 256, 0, s>>>(Nb, bverts.p, u1.p, xb.p);
    SPX_LAUNCH_CHECK();
    k_dense_gemv<TV><<<grid_for(Nb * 32, 256), 256, 0, s>>>(Nb, Bdense.p, xb.p, bverts.p, u1.p, phi.p, gB.p);
    SPX_LAUNCH_CHECK();
    prof.launches[PC_BND] += 2;
  } else if (opt.backend == 2) {
    prof.launches[PC_BND] += block_boundary_apply<TV, TM>(blk, Nb, bverts.p, u1.p, xb.p, phi.p, gB.p, s);
  } else {
    H.apply_gather<TV>(u1.p, bverts.p, phi.p, u1.p, gB.p, s);
    prof.launches[PC_BND] += H.n_far > 0 ? 3 : 2;
  }
  prof.mark(PC_BND, s);
  if (NI > 0) {
    prof.mark(PC_U2RHS, s);
    k_u2rhs<TV><<<grid_for(PIB.nslices * 32, threads), threads, 0, s>>>(NI, PIB.nslices, PIB.slice_ptr.p,
                                                                          PIB.col.p, AIB.p, gB.p, bI.p);
    SPX_LAUNCH_CHECK();
    prof.mark(PC_U2RHS, s);
    prof.launches[PC_U2RHS] += 1;
    // ||b|| of the reference's full u2 system includes the boundary rows (b[bnd] = g);
    // the interior test is slightly stricter, which only tightens the solve.
    prof.mark(PC_CG2, s);
    last2 = cg2.template solve<TV>(bI.p, xI.p, opt.rtol_u2, opt.atol, opt.maxit_u2, warm, false, sl, s,
                                   sync_stats, kind);
    prof.mark(PC_CG2, s);
    prof.launches[PC_CG2] += 1 + (sl >= 0 && cg2.hcount[sl] > 1 ? 1 : 0);
    prof.mark(PC_PHI, s);
    k_phi_interior<TV><<<grid_for(NI, 256), 256, 0, s>>>(NI, interior.p, u1.p, xI.p, phi.p);
    SPX_LAUNCH_CHECK();
    prof.mark(PC_PHI, s);
    prof.launches[PC_PHI] += 1;
  }
  ++applies;
  ++epoch;
}

template <class TV, class TM>
void DemagCtx<TV, TM>::field(TV* Hout, cudaStream_t s) {
  k_grad<TV, TM><<<grid_for(P.nslices * 32, 256), 256, 0, s>>>(N, P.nslices, P.slice_ptr.p, P.col.p, Gv.p, P.len,
                                                               phi.p, Hout);
  SPX_LAUNCH_CHECK();
}

template <class TV, class TM>
int64_t DemagCtx<TV, TM>::device_bytes() const {
  int64_t tot = 0;
  tot += P.slice_ptr.bytes() + P.col.bytes() + Div.bytes() + Dsum.bytes() + Gv.bytes() + vol.bytes();
  tot += cg1.vals.bytes() + cg1.vals64.bytes() + cg1.work.bytes() + cg1.P.col.bytes() + cg1.amg_work.bytes();
  if (cg1.amg) tot += cg1.amg->device_bytes() + cg1.amg_a32.bytes() + cg1.amg_rsum.bytes();
  tot += cg2.vals.bytes() + cg2.vals64.bytes() + cg2.work.bytes() + cg2.P.col.bytes();
  tot += AIB.bytes() + PIB.col.bytes() + Bdense.bytes();
  tot += H.device_bytes() + blk.device_bytes();
  return tot;
}

template struct DemagCtx<double, double>;
template struct DemagCtx<float, float>;
template struct DemagCtx<double, float>;

}  // namespace spx
