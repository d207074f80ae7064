// FEM operators, persistent CG solvers and the FEM/BEM demag pipeline on the device.
//
// Pipeline per call (DemagFieldLindholmGPU.compute_vec, gpu/fields/Demag_Lindholm_GPU.py:643-670):
//   b  = Ms int grad v . m                      k_div   (difference form)
//   u1 : A u1 = b - mean(b), u1 -= mean(u1)     k_cg  (:569-582; PETSc CG+GAMG there)
//   g  = B u1|bnd                               dense GEMV or H-matrix (:585-616)
//   u2 : A_II u_I = -A_IB g, u2|bnd = g          k_u2rhs + k_cg  (:618-640)
//   phi = u1 + u2 ;  H = G phi / V_i            k_grad  (:659-670)
// The Dirichlet problem is solved on the interior unknowns only; DOLFINx's identity rows for
// the boundary dofs (assemble_matrix with bcs) give the same interior solution.  CG stops when
// ||r||_2 <= max(rtol ||b||_2, atol) (unpreconditioned residual, the KSP default test with a
// zero initial guess) or after maxit.
//
// Persistent solvers: one launch per solve (krylov.cuh: one CTA, one cluster or the cooperative
// grid).  Each reduction sums its partials in the same order everywhere (deterministic, no
// contended atomics).  Every wait on memory is bounded.
#include <algorithm>
#include <cmath>

#include "fem.cuh"
#include "krylov.cuh"

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

// The entries of a row in batches of U: the batch's columns c_[] are loaded together, then the body
// gathers and loads its values for all of them before it adds them up in order, so a row's chain is
// one column load and one gather per batch instead of per entry.  Batch sizes by measurement
// (registers against warps in flight): k_div 3, 400x400x2 film 39 -> 34 us, 64 boxes of 2,646 nodes
// 34 -> 28 us, one box 6.6 -> 3.9 us (four: 36, 31, 4.2; eight: 76 us on the boxes); k_grad 4, one
// box 6.0 -> 3.8 us; k_u2rhs 8, 10.5 -> 5 us on the film and the boxes, one box 4.2 -> 2.1 us.
// k0_: first entry of the batch, i0_: its position.
#define SELL_BATCHES(U, width, ...)                                                            \
  for (int k0_ = 0; k0_ < (width); k0_ += U) {                                                 \
    const int64_t i0_ = base_ + ((int64_t)k0_ << 5) + lane_;                                   \
    int32_t c_[U];                                                                             \
    _Pragma("unroll") for (int u = 0; u < U; ++u) c_[u] = k0_ + u < (width) ? col[i0_ + 32 * u] : 0; \
    __VA_ARGS__                                                                                \
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
      SELL_BATCHES(3, width, {
        TV x[3], y[3], z[3];
        TM d0[3], d1[3], d2[3];
        _Pragma("unroll") for (int u = 0; u < 3; ++u) if (k0_ + u < width) {
          const int64_t j = c_[u], idx = i0_ + 32 * u;
          x[u] = m[3 * j];
          y[u] = m[3 * j + 1];
          z[u] = m[3 * j + 2];
          d0[u] = D[idx];
          d1[u] = D[L + idx];
          d2[u] = D[2 * L + idx];
        }
        _Pragma("unroll") for (int u = 0; u < 3; ++u) if (k0_ + u < width)
          acc += static_cast<TV>(d0[u]) * (x[u] - mx) + static_cast<TV>(d1[u]) * (y[u] - my) +
                 static_cast<TV>(d2[u]) * (z[u] - mz);
      })
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
      SELL_BATCHES(4, width, {
        TV p[4];
        TM g0[4], g1[4], g2[4];
        _Pragma("unroll") for (int u = 0; u < 4; ++u) if (k0_ + u < width) {
          const int64_t idx = i0_ + 32 * u;
          p[u] = phi[c_[u]];
          g0[u] = Gv[idx];
          g1[u] = Gv[L + idx];
          g2[u] = Gv[2 * L + idx];
        }
        _Pragma("unroll") for (int u = 0; u < 4; ++u) if (k0_ + u < width) {
          const TV q = p[u] - pi;
          hx += static_cast<TV>(g0[u]) * q;
          hy += static_cast<TV>(g1[u]) * q;
          hz += static_cast<TV>(g2[u]) * q;
        }
      })
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
      SELL_BATCHES(8, width, {
        double x[8];
        double w[8];
        _Pragma("unroll") for (int u = 0; u < 8; ++u) if (k0_ + u < width) {
          x[u] = static_cast<double>(g[c_[u]]);
          w[u] = v[i0_ + 32 * u];
        }
        _Pragma("unroll") for (int u = 0; u < 8; ++u) if (k0_ + u < width) acc += w[u] * x[u];
      })
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

// ------------------------------------------------------------------ CG with FP64 refinement
// The scaled system D^-1/2 A D^-1/2 (unit diagonal) by CG in TM (FP32 or FP64) inside FP64
// iterative refinement, Chronopoulos and Gear's form of CG (both dot products of an iteration in
// one reduction).
//
// What bounds it: a solve takes tens of iterations of 10^3 to 10^5 rows, so the barriers and
// the load chain between them, not bytes.  The matrix stays in shared memory for the solve (but on
// the largest systems).
//   * A system whose matrix and vectors fit the shared memory of one CTA, or of a cluster of up
//     to eight, runs there: hardware barriers (40 and 450 cycles against 2,600 over the grid), an
//     update and a product phase per iteration, the residual gathered from (distributed) shared
//     memory, the columns kept as its 32-bit addresses.  Bound by shared-memory bandwidth.
//   * Larger ones run on the grid, one phase per iteration: instead of updating r and q, waiting,
//     and multiplying, every row forms its neighbours' new residuals itself,
//       r_j' = r_j - alpha (s_j + beta q_j),   s_i' = sum_j a_ij r_j',
//     from the records {r, s, q} of the last phase (one 16-byte FP32 gather per entry, two
//     buffers), which saves one of two grid barriers.
//   * Where the records' bytes cost more than the barrier, on the grid in two phases again, with
//     plain vectors (four or eight bytes per gather, most of them in the L1 cache, which no
//     matrix takes) and twice the warps.  1.03 million nodes off the lattice: FP32 43 us an iteration
//     (120 with records, whose matrix streams through L2), FP64 59 (160).
constexpr int CG_BLOCK = 512;
constexpr int CG_BLOCK_LARGE = 1024;  // TEAM_GRID_LARGE
constexpr int CG_DYN_MAX = 220 * 1024;
constexpr int CG_SLICES_PER_CTA = 16;  // CTAs of a cluster: one per 16 slices (a round of its warps)
// Where TEAM_GRID is the faster form on the grid, by the entries and slices of a CTA: in FP32 as far
// as its shared memory holds the matrix and its 16 warps go over five rounds of slices, in FP64 (records
// of 32 bytes) for fewer entries.  us per iteration with TEAM_GRID / TEAM_GRID_LARGE by 10^3 entries and
// slices of a CTA: FP32 8 and 15 5.3 / 7.5, 15 and 32 6.5 / 7.8, 23 and 48 8.1 / 9.8 (nodes off the lattice, 15
// entries a row); 11 and 48 6.7 / 8.7, 17 and 76 8.7 / 10.5, 16 and 72 9.8 / 9.9, 19 and 86 11.3 / 9.8, 25 and 113
// 13.9 / 12.3 (on it, 7 entries a row).  FP64 8 k 7.0 / 8.2, 10 k 9.5 / 8.1, 15 k 12.4 / 8.6 (off the lattice);
// 7 k 6.9 / 7.5, 11 k 8.8 / 9.3, 17 k 12.5 / 11.7 (on it).
template <class TM>
constexpr int64_t cg_record_entries() {
  return sizeof(TM) == sizeof(float) ? 27000 : 8000;
}
constexpr int64_t CG_RECORD_SLICES = 80;
static_assert(27000 * 8 + (CG_RECORD_SLICES + 8) * 4 <= CG_DYN_MAX, "entries and slice bounds of a CTA");

extern __shared__ __align__(16) unsigned char cg_smem[];

template <class TM> struct CgRec;  // r, s, q of one row
template <> struct CgRec<float> {
  float r, s, q;
  using Store = float4;
  static __device__ __forceinline__ CgRec load(const Store* p) {
    const float4 v = *p;
    return {v.x, v.y, v.z};
  }
  __device__ __forceinline__ void store(Store* p) const { *p = make_float4(r, s, q, 0.0f); }
};
struct __align__(32) CgRecD { double r, s, q, pad; };
template <> struct CgRec<double> {
  double r, s, q;
  using Store = CgRecD;
  static __device__ __forceinline__ CgRec load(const Store* p) {
    const double2 a = *reinterpret_cast<const double2*>(p);
    return {a.x, a.y, p->q};
  }
  __device__ __forceinline__ void store(Store* p) const {
    *reinterpret_cast<double2*>(p) = make_double2(r, s);
    p->q = q;
  }
};

constexpr int CG_SMEM_VECS = 5;  // r, s, q, p, d of a CTA's rows in shared memory (CTA and cluster teams)

template <class TV, class TM>
struct CgParams {
  int64_t n, nslices;
  const int64_t* sp;
  const int32_t* col;
  const TM* val;
  const double* v64;
  const double* sdinv;
  const double* diag;
  const TV* b;
  TV* x;
  double *bh, *y;
  TM *p, *d, *r, *s, *q;  // r, s, q: TEAM_GRID_LARGE; in records g0, g1: TEAM_GRID
  typename CgRec<TM>::Store *g0, *g1;
  double* part;
  unsigned int* bar;
  int* err;
  int* iters;
  double* resid;
  unsigned long long* iters_acc;
  double* res_acc;  // [0] sum of initial relative residuals, [1] sum of final ones
  double rtol, atol, inner_rtol;
  int maxit, max_outer, warm, project;
  int bh_given;     // bh already holds the scaled, projected right-hand side (FP64)
  int32_t off_cap;  // slice bounds kept in shared memory (none by TEAM_GRID_LARGE)
  int32_t cap;      // entries kept in shared memory per CTA
  int32_t rows;     // rows of the largest block (CTA and cluster teams)
};

template <class TV, class TM, int TEAM>
__global__ void __launch_bounds__(TEAM == TEAM_GRID_LARGE ? CG_BLOCK_LARGE : CG_BLOCK, 1) k_cg(const __grid_constant__ CgParams<TV, TM> P) {
  using Rec = CgRec<TM>;
  constexpr bool SM = TEAM == TEAM_CTA || TEAM == TEAM_CLUSTER;  // vectors in shared memory
  constexpr bool REC = TEAM == TEAM_GRID;                        // r, s, q in records
  constexpr bool LARGE = TEAM == TEAM_GRID_LARGE;                // nothing in shared memory
  constexpr int U = sizeof(TM) == 4 ? 8 : 4;  // records in flight per row (grid)
  __shared__ TeamShared S;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int64_t n = P.n;
  if (TEAM == TEAM_CLUSTER) cluster_sync_all();  // every CTA runs before the first remote store
  // this CTA's block of slices; bounds, values and columns in shared memory (not LARGE)
  const int64_t s0 = P.nslices * blockIdx.x / gridDim.x;
  const int cnt = static_cast<int>(P.nslices * (blockIdx.x + 1) / gridDim.x - s0);
  const int64_t base = P.sp[s0];
  int32_t* soff = reinterpret_cast<int32_t*>(cg_smem);
  TM* sval = reinterpret_cast<TM*>(cg_smem + static_cast<size_t>(P.off_cap) * 4);
  int32_t* scol = reinterpret_cast<int32_t*>(sval + P.cap);
  TM* vr = reinterpret_cast<TM*>(scol + P.cap);
  TM *vs = vr + P.rows, *vq = vs + P.rows, *vp = vq + P.rows, *vd = vp + P.rows;
  const unsigned ar = static_cast<unsigned>(__cvta_generic_to_shared(vr));
  if constexpr (LARGE) {
    vr = P.r; vs = P.s; vq = P.q; vp = P.p; vd = P.d;
  } else {
    for (int k = threadIdx.x; k <= cnt; k += blockDim.x) soff[k] = static_cast<int32_t>(P.sp[s0 + k] - base);
    __syncthreads();
    const int m = soff[cnt];
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
      sval[k] = P.val[base + k];
      int32_t c = P.col[base + k];
      if (SM) {  // the address of the column's residual in its owner's shared memory
        const int64_t own = ((static_cast<int64_t>(c >> 5) + 1) * gridDim.x - 1) / P.nslices;
        const unsigned a = ar + static_cast<unsigned>(c - 32 * (P.nslices * own / gridDim.x)) * sizeof(TM);
        c = static_cast<int32_t>(TEAM == TEAM_CLUSTER ? cluster_addr(a, static_cast<unsigned>(own)) : a);
      }
      scol[k] = c;
    }
    __syncthreads();
  }
  auto bounds = [&](int k, int64_t& o, int& width) {
    if constexpr (LARGE) {
      const int64_t a = P.sp[s0 + k];
      o = a - base;
      width = static_cast<int>((P.sp[s0 + k + 1] - a) >> 5);
    } else {
      o = soff[k];
      width = (soff[k + 1] - soff[k]) >> 5;
    }
  };
#define CG_ROWS_BEGIN                       \
  for (int k = wid; k < cnt; k += nw) {     \
    const int64_t i = (s0 + k) * 32 + lane; \
    if (i < n) {
#define CG_ROWS_END \
  }                 \
  }
  int flip = 0;
  auto sum2 = [&](double& a, double& b) { return team_sum<TEAM>(S, P.part, P.bar, P.err, flip, a, b); };
  double meanb = 0.0, dummy = 0.0;
  if (P.project && !P.bh_given) {
    double part = 0.0;
    CG_ROWS_BEGIN part += static_cast<double>(P.b[i]);
    CG_ROWS_END
    if (!sum2(part, dummy)) return;
    meanb = part / static_cast<double>(n);
  }
  double bb = 0.0, rho = 0.0, rho0 = -1.0, tol2 = 0.0;
  bool zero = !P.warm;  // y = 0
  int total = 0, outers = 0;
  for (int outer = 0;; ++outer) {
    ++outers;
    // true residual in FP64 (and, the first time, the right-hand side); start of the inner solve.
    // After the last of max_outer inner solves too: the residual reported is that of the solution.
    {
      double rh = 0.0, b2 = 0.0;
      CG_ROWS_BEGIN
        const double sd = P.sdinv[i], dg = P.diag[i];
        double r64;
        if (outer == 0 && !P.bh_given) {
          const double bv = static_cast<double>(P.b[i]) - meanb;
          r64 = bv * sd;
          P.bh[i] = r64;
          b2 += bv * bv;
        } else {
          r64 = P.bh[i];
          if (outer == 0) {
            const double bv = r64 / sd;
            b2 += bv * bv;
          }
        }
        if (zero) {
          P.y[i] = 0.0;
        } else {
          int64_t o;
          int width;
          bounds(k, o, width);
          const double* gv = P.v64 + base + o + lane;
          const int32_t* gc = P.col + base + o + lane;
          double acc = 0.0, acc2 = 0.0;
          for (int j = 0; j < width; j += 4) {
            double w[4], g[4];
            int32_t c[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const bool in = j + u < width;
              c[u] = in ? gc[(j + u) * 32] : 0;
              w[u] = in ? gv[(j + u) * 32] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) g[u] = j + u < width ? P.y[c[u]] : 0.0;
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
              acc += w[u] * g[u];
              acc2 += w[u + 1] * g[u + 1];
            }
          }
          r64 -= acc + acc2;
        }
        rh += dg * r64 * r64;
        if constexpr (!REC) {
          const int64_t row = SM ? 32 * k + lane : i;
          vr[row] = static_cast<TM>(r64);
          vs[row] = vq[row] = vp[row] = vd[row] = TM(0);
        } else {
          Rec{static_cast<TM>(r64), TM(0), TM(0)}.store(P.g0 + i);
          P.p[i] = TM(0);
          P.d[i] = TM(0);
        }
      CG_ROWS_END
      if (!sum2(rh, b2)) return;
      rho = rh;
      if (outer == 0) {
        bb = b2;
        tol2 = fmax(P.rtol * P.rtol * bb, P.atol * P.atol);
        if (!(bb > 0.0)) {  // b = 0: the solution is 0 (a warm start would only chase rounding noise)
          CG_ROWS_BEGIN P.y[i] = 0.0;
          CG_ROWS_END
          rho = rho0 = 0.0;
          break;
        }
      }
    }
    zero = false;
    if (rho0 < 0.0) rho0 = rho;
    if (rho <= tol2 || total >= P.maxit || outer == P.max_outer) break;
    // reduce the residual only as far as the target needs (with a 0.3 margin), at most
    // by inner_rtol per refinement step (the inner solve's reliable range)
    const double need = 0.3 * sqrt(tol2 / rho);
    const double itol = fmax(P.inner_rtol, fmin(need, 0.5));
    // alpha = gm / den, den = dl - beta^2 den_prev (= dl - beta gm / alpha_prev): one division
    // between the sums and the next phase; 1 / gm is formed while they are on their way
    double g0 = 0.0, ginv = 0.0, den = 0.0;
    TM a = TM(0), bt = TM(0);
    for (int it = -1;; ++it) {  // it = -1 (a = bt = 0) only multiplies: s = A r
      double gm = 0.0, dl = 0.0;
      if constexpr (!REC) {
        if (it >= 0) {
          CG_ROWS_BEGIN
            const int64_t row = SM ? 32 * k + lane : i;
            const TM qn = vs[row] + bt * vq[row], pn = vr[row] + bt * vp[row];
            vq[row] = qn;
            vp[row] = pn;
            vd[row] += a * pn;
            vr[row] -= a * qn;
          CG_ROWS_END
          if (!team_barrier<TEAM>(P.bar, P.err)) return;
        }
        CG_ROWS_BEGIN
          const int64_t row = SM ? 32 * k + lane : i;
          int64_t o;
          int width;
          bounds(k, o, width);
          TM acc = TM(0), acc2 = TM(0);
          if constexpr (SM) {
            const int so = static_cast<int>(o) + lane;
            for (int j = 0; j < width; j += 8) {
              unsigned c[8];
              TM g[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) c[u] = j + u < width ? static_cast<unsigned>(scol[so + (j + u) * 32]) : ar;
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (j + u < width) g[u] = team_load<TEAM>(c[u], TM(0));
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (j + u < width) {
                  if (u & 1) acc2 += sval[so + (j + u) * 32] * g[u];
                  else acc += sval[so + (j + u) * 32] * g[u];
                }
            }
          } else {
            const TM* gv = P.val + base + o + lane;
            const int32_t* gc = P.col + base + o + lane;
            for (int j = 0; j < width; j += 8) {
              int32_t c[8];
              TM w[8], g[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                const bool in = j + u < width;
                c[u] = in ? gc[(j + u) * 32] : 0;
                w[u] = in ? gv[(j + u) * 32] : TM(0);
              }
#pragma unroll
              for (int u = 0; u < 8; ++u) g[u] = j + u < width ? vr[c[u]] : TM(0);
#pragma unroll
              for (int u = 0; u < 8; u += 2) {
                acc += w[u] * g[u];
                acc2 += w[u + 1] * g[u + 1];
              }
            }
          }
          const TM sn = acc + acc2;
          vs[row] = sn;
          const double rd = static_cast<double>(vr[row]);
          gm += rd * rd;
          dl += rd * static_cast<double>(sn);
        CG_ROWS_END
      } else {
        const typename Rec::Store* cur = (it & 1) ? P.g0 : P.g1;
        typename Rec::Store* nxt = (it & 1) ? P.g1 : P.g0;
        CG_ROWS_BEGIN
          const Rec me = Rec::load(cur + i);
          const TM pold = P.p[i], dold = P.d[i];
          int64_t o;
          int width;
          bounds(k, o, width);
          TM acc = TM(0), acc2 = TM(0);
          const int so = static_cast<int>(o) + lane;
          for (int j = 0; j < width; j += U) {
            int32_t c[U];
            Rec g[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
              c[u] = j + u < width ? scol[so + (j + u) * 32] : 0;
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (j + u < width) g[u] = Rec::load(cur + c[u]);
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (j + u < width) {
                const TM w = sval[so + (j + u) * 32];
                const TM rj = g[u].r - a * (g[u].s + bt * g[u].q);
                if (u & 1) acc2 += w * rj; else acc += w * rj;
              }
          }
          const TM qn = me.s + bt * me.q, pn = me.r + bt * pold, rn = me.r - a * qn, sn = acc + acc2;
          Rec{rn, sn, qn}.store(nxt + i);
          P.p[i] = pn;
          P.d[i] = dold + a * pn;
          const double rd = static_cast<double>(rn);
          gm += rd * rd;
          dl += rd * static_cast<double>(sn);
        CG_ROWS_END
      }
      if (!sum2(gm, dl)) return;
      if (it < 0) g0 = gm; else ++total;
      if (gm <= itol * itol * g0 || total >= P.maxit || !(gm > 0.0) || !(dl > 0.0)) break;
      const double beta = gm * ginv;  // 0 on the first step
      den = dl - beta * beta * den;
      if (!(den > 0.0)) break;  // lost to rounding: the next refinement starts from the true residual
      bt = static_cast<TM>(beta);
      // the quotient in FP64, then rounded: gm and den are squares of the residual's norm and leave
      // the range of FP32 (1e-38) long before the residual does
      a = static_cast<TM>(gm / den);
      ginv = 1.0 / gm;
    }
    CG_ROWS_BEGIN
      P.y[i] += static_cast<double>(SM ? vd[32 * k + lane] : P.d[i]);
    CG_ROWS_END
    if (!team_barrier<TEAM>(P.bar, P.err)) return;
  }
  double mx = 0.0;
  if (P.project) {
    double sx = 0.0;
    CG_ROWS_BEGIN sx += P.y[i] * P.sdinv[i];
    CG_ROWS_END
    dummy = 0.0;
    if (!sum2(sx, dummy)) return;
    mx = sx / static_cast<double>(n);
  }
  CG_ROWS_BEGIN
    const double sd = P.sdinv[i];
    const double xv = P.y[i] * sd - mx;
    P.x[i] = static_cast<TV>(xv);
    if (P.project) P.y[i] = xv / sd;
  CG_ROWS_END
#undef CG_ROWS_BEGIN
#undef CG_ROWS_END
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

template <class TV, class TM>
const void* cg_kernel(int team) {
  return team == TEAM_CTA ? reinterpret_cast<const void*>(k_cg<TV, TM, TEAM_CTA>)
         : team == TEAM_CLUSTER ? reinterpret_cast<const void*>(k_cg<TV, TM, TEAM_CLUSTER>)
         : team == TEAM_GRID    ? reinterpret_cast<const void*>(k_cg<TV, TM, TEAM_GRID>)
                                : reinterpret_cast<const void*>(k_cg<TV, TM, TEAM_GRID_LARGE>);
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
  if (sizeof(TM) == sizeof(float)) vals64.upload(v64);
  y64.alloc(n);
  y64.zero();
  bh64.alloc(n);
  work.alloc(static_cast<size_t>(n) * (2 * sizeof(TM) + 2 * sizeof(typename CgRec<TM>::Store)));
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
  // the team of k_cg: one CTA or a cluster when matrix and vectors fit their shared memory, else
  // the grid, a slice a warp.  Per iteration (before: a grid kernel with one or two phases, own
  // vectors and matrix in global memory): 11 slices on one CTA 1.3 us, 46 slices (20x20x5 box) on
  // four 1.8 us (10 us on its two CTAs before; 2.3 on eight, 3.0 on two), 132 slices on eight
  // 2.9 us (grid 4.7), 428 slices on eight 4.5 us (grid 4.5); the grid 4.4-5.2 us up to 1,600 slices (FP32)
  int64_t cnt = 0, need = 0;  // slices and entries of the largest block
  const int64_t eb = sizeof(TM) + sizeof(int32_t);
  auto blocks = [&](int g) {
    grid = g;
    cnt = need = 0;
    for (int c = 0; c < g; ++c) {
      const int64_t a = s.nslices * c / g, e = s.nslices * (c + 1) / g;
      cnt = std::max(cnt, e - a);
      need = std::max(need, s.slice_ptr[e] - s.slice_ptr[a]);
    }
    off_cap = static_cast<int32_t>((cnt + 1 + 3) / 4 * 4);
  };
  auto small_bytes = [&] { return off_cap * 4 + need * eb + cnt * 32 * CG_SMEM_VECS * static_cast<int64_t>(sizeof(TM)); };
  int g = 1;
  while (g < TEAM_MAX_CLUSTER && s.nslices > static_cast<int64_t>(g) * CG_SLICES_PER_CTA) g *= 2;
  blocks(g);
  while (g < TEAM_MAX_CLUSTER && small_bytes() > CG_DYN_MAX) blocks(g *= 2);
  if (small_bytes() <= CG_DYN_MAX) {
    team = g == 1 ? TEAM_CTA : TEAM_CLUSTER;
    cap = static_cast<int32_t>(need);
    rows = static_cast<int32_t>(cnt * 32);
    smem_bytes = static_cast<size_t>(small_bytes());
    threads = 32 * static_cast<int>(std::min<int64_t>(CG_BLOCK / 32, std::max<int64_t>(cnt, 4)));
  } else {
    auto grid_blocks = [&](int t) {
      threads = t;
      blocks(static_cast<int>(std::min<int64_t>((s.nslices + t / 32 - 1) / (t / 32), num_sms(dev))));
    };
    team = TEAM_GRID;
    grid_blocks(CG_BLOCK);
    rows = 0;
    if (need <= cg_record_entries<TM>() && cnt <= CG_RECORD_SLICES) {
      cap = static_cast<int32_t>(need);
      smem_bytes = static_cast<size_t>(off_cap * 4 + need * eb);
    } else {
      team = TEAM_GRID_LARGE;
      grid_blocks(CG_BLOCK_LARGE);
      off_cap = cap = 0;
      smem_bytes = 0;
      // hundreds of iterations a solve, which every refinement starts anew: in FP64 one run as far as
      // its recurrence holds (to 1e-9 on 202,005 nodes 1,448 -> 1,200 iterations, 15.4 -> 12.9 ms)
      if (sizeof(TM) == sizeof(double)) inner_rtol = 1e-12;
    }
  }
  part.alloc(4 * 4 * static_cast<size_t>(std::max(grid, num_sms(dev))));
  std::vector<const void*> ks{cg_kernel<double, TM>(team)};
  if constexpr (sizeof(TM) == sizeof(float)) ks.push_back(cg_kernel<float, TM>(team));
  if (team != TEAM_GRID_LARGE)
    for (const void* k : ks) SPX_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, CG_DYN_MAX));
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
  SPX_CHECK(sizeof(TM) == sizeof(float) || sizeof(TV) == sizeof(double), "FP64 CG needs FP64 vectors");
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
      double* target = y64.p;
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
  if (seg) {
    k_seg_center_bh<TV><<<sgrid, 256, 0, st>>>(seg_off.p, seg_maxch, seg_part.p, b, seg_sd, bh64.p);
    SPX_LAUNCH_CHECK();
  }
  if (use_amg) {
    launch_amg<TV>(b, x, rtol, atol, maxit, warm, project, st, seg);
  } else {
    CgParams<TV, TM> q;
    q.n = n; q.nslices = P.nslices; q.sp = P.slice_ptr.p; q.col = P.col.p;
    q.val = vals.p; q.sdinv = sdinv64.p; q.diag = diag64.p;
    q.v64 = sizeof(TM) == sizeof(float) ? vals64.p : reinterpret_cast<const double*>(vals.p);
    q.b = b; q.x = x;
    q.bh = bh64.p; q.y = y64.p;
    using Store = typename CgRec<TM>::Store;
    q.g0 = reinterpret_cast<Store*>(work.p);
    q.g1 = q.g0 + n;
    q.p = reinterpret_cast<TM*>(q.g1 + n);
    q.d = q.p + n;
    q.r = reinterpret_cast<TM*>(work.p);  // in place of the records
    q.s = q.r + n;
    q.q = q.s + n;
    q.part = part.p; q.bar = bar.p; q.err = err.p; q.iters = iters.p; q.resid = resid.p;
    q.iters_acc = iters_acc.p;
    q.res_acc = res_acc.p;
    q.rtol = rtol; q.atol = atol; q.inner_rtol = inner_rtol;
    q.maxit = maxit; q.max_outer = max_outer; q.warm = warm ? 1 : 0;
    q.bh_given = seg ? 1 : 0;
    q.project = project ? 1 : 0;
    q.off_cap = off_cap;
    q.cap = cap;
    q.rows = rows;
    const void* k = cg_kernel<TV, TM>(team);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    if (team == TEAM_CLUSTER) {
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = grid;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    } else {
      at[0].id = cudaLaunchAttributeCooperative;
      at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void* args[] = {&q};
    SPX_CUDA(cudaLaunchKernelExC(&cfg, k, args));
  }
  if (project && seg_off.n > 1) {
    k_seg_sum<TV><<<sgrid, 256, 0, st>>>(seg_off.p, seg_maxch, x, y64.p, seg_sd, seg_part.p);
    SPX_LAUNCH_CHECK();
    k_seg_center<TV><<<sgrid, 256, 0, st>>>(seg_off.p, seg_maxch, seg_part.p, x, y64.p, seg_sd);
    SPX_LAUNCH_CHECK();
  }
  if (slot == 0 && stage_correct && have_pred0) {  // stage 1's prediction error
    if (!delta.n) delta.alloc(n);
    k_axpy_sub<<<grid_for(n, 256), 256, 0, st>>>(n, y64.p, pred0.p, delta.p, 0);
    SPX_LAUNCH_CHECK();
    have_delta = true;
    have_pred0 = false;
  }
  if (slot >= 0) {
    double* dst = hist[slot][hhead[slot]].p;
    const double* src = y64.p;
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
