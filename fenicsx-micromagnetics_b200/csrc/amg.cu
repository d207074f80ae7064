// Device side of the smoothed-aggregation AMG (amg.cuh): level upload, the FP32 V-cycle
// and the FP64 preconditioned CG that uses it, in one persistent cooperative kernel.
//
// Level layout: A_l and P_l are SELL-32 (one thread per row, 32 rows per slice, padding
// entries point at column 0 with value 0); R_l = P_l^T is CSR swept by `r_lanes` lanes per
// row (its rows are long); FP32 values; FP32 vectors b, D^-1 b, x, x2, d, r per level.  Every
// phase is swept by the whole grid with a grid barrier after it; the dense coarsest level
// (at most a few thousand unknowns) is one GEMV with its precomputed inverse, a warp per row.
//
// PCG (FP64 vectors, on A itself; in exact arithmetic the same iterates as on D^-1/2 A D^-1/2):
//   u = V(r);  beta = (r,u)/(r,u)_old;  c = (d,u)/(1,d) (singular systems: remove the constant
//   from u, d the diagonal);  p = u - c + beta p;
//   q = A u + beta q  (A 1 = 0, so q = A p without a second SpMV), with A u evaluated as
//   sum_j a_ij (u_j - u_i) + (sum_j a_ij) u_i, FP32 a_ij (those of the cycle), FP64 sums;
//   alpha = (r,u)/(p,q);  y += alpha p;  r -= alpha q.
// The recurrence residual is confirmed against the true FP64 residual (FP64 values) before
// returning; stopping rule ||b - A x|| <= max(rtol ||b||, atol).
//
// What bounds k_pcg_amg is the chain of loads inside each of its 15 or so phases per
// iteration, not bytes: 148 CTAs sweep 10^3 to 10^6 rows between two grid barriers of 1.3 us.
// So (1) every CTA owns a contiguous block of slices of each level, and keeps their values,
// columns and slice bounds in shared memory for the whole solve, as far as 220 KB go (finest
// level first, which five phases of an iteration read): a phase's chain is one gather, and no
// matrix byte crosses L2 again; slices past that stream from global memory in the same loop;
// (2) eight gathers of a row are in flight; (3) the level descriptors are kernel parameters;
// (4) the sums of the PCG ride on the barrier (sync_sum).  Per iteration, against sweeps that
// read the matrices from global memory, two gathers in flight on a row's last columns:
// 183 -> 96 us on the 400x400x2 film (level-0 sweeps 12-21 -> 6-8 us, product 18 -> 9.5,
// update 13 -> 6; the restriction, the prolongation and the dense level, 9-12 us each, read
// 12-25 MB through L2), 150 -> 80 us on the union of 64 boxes (375,280 nodes), 48 -> 26 us on
// the 20x20x5 box, where a phase is 2-4 us, 1.3 of it the barrier.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "amg.cuh"
#include "fem.cuh"

namespace spx {

std::atomic<int> g_pcg_timing{0};  // phase timing marks of the AMG-PCG kernel (spx_debug_pcg_timing)

// The cycle loads the matrices of its cycled levels with an L2 evict_last policy.  A larger L2
// set-aside for persisting lines (a limit of this process's context, not a GPU setting) can be
// requested with SPX_L2_PERSIST_MB (MiB, raised only, capped by the device's maximum).  It is
// off by default: measured on the 400 x 400 x 2 film, raising it from the context's 24 MB to
// 75 MB left the u1 solve unchanged and slowed the streaming boundary apply by 7 %.
void reserve_persisting_l2(int64_t bytes, int dev) {
  const char* e = std::getenv("SPX_L2_PERSIST_MB");
  if (!e) return;
  bytes = std::atoll(e) << 20;
  if (bytes <= 0) return;
  int mx = 0;
  SPX_CUDA(cudaDeviceGetAttribute(&mx, cudaDevAttrMaxPersistingL2CacheSize, dev));
  if (mx <= 0) return;
  size_t cur = 0;
  SPX_CUDA(cudaDeviceGetLimit(&cur, cudaLimitPersistingL2CacheSize));
  const size_t want = std::min<size_t>(static_cast<size_t>(mx), static_cast<size_t>(bytes));
  if (want > cur) SPX_CUDA(cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, want));
}

namespace {

void csr_to_sell(const CsrHost& A, HostSell& s, std::vector<float>& val) {
  const int64_t n = A.n;
  s.nrows = n;
  s.nslices = (n + SELL_C - 1) / SELL_C;
  s.slice_ptr.assign(s.nslices + 1, 0);
  for (int64_t sl = 0; sl < s.nslices; ++sl) {
    int64_t w = 0;
    for (int64_t r = sl * SELL_C; r < std::min(n, (sl + 1) * SELL_C); ++r) w = std::max(w, A.rp[r + 1] - A.rp[r]);
    s.slice_ptr[sl + 1] = s.slice_ptr[sl] + w * SELL_C;
  }
  const int64_t L = s.slice_ptr.back();
  s.col.assign(L, 0);
  val.assign(L, 0.0f);
  for (int64_t r = 0; r < n; ++r) {
    const int64_t sl = r / SELL_C, lane = r % SELL_C;
    int64_t q = 0;
    for (int64_t k = A.rp[r]; k < A.rp[r + 1]; ++k, ++q) {
      const int64_t pos = s.slice_ptr[sl] + q * SELL_C + lane;
      s.col[pos] = A.ci[k];
      val[pos] = static_cast<float>(A.v[k]);
    }
  }
  s.map.clear();
}

// in-place Gauss-Jordan inverse of an SPD matrix (no pivoting), one pivot per step
__global__ void k_gj_pivot(double* __restrict__ M, double* __restrict__ colk, int64_t n, int64_t k) {
  const double p = M[k * n + k];
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) colk[i] = M[i * n + k];
  __syncthreads();
  for (int64_t j = threadIdx.x; j < n; j += blockDim.x) M[k * n + j] = (j == k) ? 1.0 / p : M[k * n + j] / p;
}
__global__ void k_gj_update(double* __restrict__ M, const double* __restrict__ colk, int64_t n, int64_t k) {
  const int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (e >= n * n) return;
  const int64_t i = e / n, j = e - i * n;
  if (i == k) return;
  const double f = colk[i];
  if (j == k)
    M[e] = -f * M[k * n + k];
  else
    M[e] -= f * M[k * n + j];
}
// FP32 copy of an n x n matrix into rows of ld >= n entries (zero padded)
__global__ void k_to_float_rows(const double* __restrict__ a, float* __restrict__ b, int64_t n, int64_t ld) {
  const int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (e >= n * ld) return;
  const int64_t i = e / ld, j = e - i * ld;
  b[e] = j < n ? static_cast<float>(a[i * n + j]) : 0.0f;
}

}  // namespace

void AmgDevice::upload(const AmgHost& h, cudaStream_t s, const int64_t* sp0, const int32_t* col0, const float* val0,
                       int64_t nslices0, int nrep, int grid) {
  reps = nrep;
  nlev = static_cast<int>(h.lv.size());
  n0 = h.lv[0].A.n;
  nc = h.lv.back().A.n;
  A.clear(); P.clear(); rrp.clear(); rcol.clear();
  val.clear(); pval.clear(); rval.clear(); dinv.clear(); vec.clear();
  A.resize(nlev); P.resize(nlev); rrp.resize(nlev); rcol.resize(nlev);
  val.resize(nlev); pval.resize(nlev); rval.resize(nlev); dinv.resize(nlev); vec.resize(nlev);
  sizes.assign(nlev, 0);
  nnz.assign(nlev, 0);
  pnnz.assign(nlev, 0);
  rnnz.assign(nlev, 0);
  SPX_CHECK(nlev <= AMG_MAX_LEVELS, "too many AMG levels");
  std::vector<AmgLevelDev>& d = lv;
  d.assign(nlev, AmgLevelDev{});
  need.assign(nlev, 0);
  cnt.assign(nlev, 0);
  res.assign(nlev, AmgResident{-1, 0, 0, 0, 0, 0});
  for (int l = 0; l < nlev; ++l) {
    const AmgHostLevel& L = h.lv[l];
    sizes[l] = L.A.n;
    nnz[l] = static_cast<int64_t>(L.A.ci.size());
    pnnz[l] = static_cast<int64_t>(L.P.ci.size());
    rnnz[l] = static_cast<int64_t>(L.R.ci.size());
    AmgLevelDev& D = d[l];
    std::memset(&D, 0, sizeof(D));
    D.n = L.A.n;
    std::vector<float> di(L.dinv.begin(), L.dinv.end());
    dinv[l].upload(di, s);
    D.dinv = dinv[l].p;
    const int64_t nv = L.A.n * reps;  // every level vector holds the reps blocks one after the other
    vec[l].alloc(6 * static_cast<size_t>(nv));
    vec[l].zero(s);
    D.b = vec[l].p;
    D.db = vec[l].p + nv;
    D.x = vec[l].p + 2 * nv;
    D.x2 = vec[l].p + 3 * nv;
    D.d = vec[l].p + 4 * nv;
    D.r = vec[l].p + 5 * nv;
    if (l + 1 == nlev) break;  // dense coarsest: vectors only
    HostSell hs, hp;
    std::vector<float> v, vp;
    std::vector<int64_t> sph;
    if (l == 0 && sp0) {
      D.nslices = nslices0;
      D.sp = sp0;
      D.col = col0;
      D.val = val0;
      sph.resize(nslices0 + 1);
      SPX_CUDA(cudaMemcpyAsync(sph.data(), sp0, sph.size() * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
      SPX_CUDA(cudaStreamSynchronize(s));
    } else {
      csr_to_sell(L.A, hs, v);
      A[l].upload(hs, s);
      val[l].upload(v, s);
      D.nslices = hs.nslices;
      D.sp = A[l].slice_ptr.p;
      D.col = A[l].col.p;
      D.val = val[l].p;
      sph = hs.slice_ptr;
    }
    // slices and entries of the largest CTA block of this level (slices [ns c / G, ns (c+1) / G))
    for (int c = 0; c < grid; ++c) {
      const int64_t a = D.nslices * c / grid, e = D.nslices * (c + 1) / grid;
      cnt[l] = std::max(cnt[l], e - a);
      need[l] = std::max(need[l], sph[e] - sph[a]);
    }
    csr_to_sell(L.P, hp, vp);
    P[l].upload(hp, s);
    pval[l].upload(vp, s);
    D.p_nslices = hp.nslices;
    D.p_sp = P[l].slice_ptr.p;
    D.p_col = P[l].col.p;
    D.p_val = pval[l].p;
    rrp[l].upload(L.R.rp, s);
    rcol[l].upload(L.R.ci, s);
    std::vector<float> vr(L.R.v.begin(), L.R.v.end());
    rval[l].upload(vr, s);
    D.r_rp = rrp[l].p;
    D.r_col = rcol[l].p;
    D.r_val = rval[l].p;
    const double avg = static_cast<double>(L.R.ci.size()) / std::max<int64_t>(L.R.n, 1);
    int lanes = 1;  // about eight entries per lane
    while (lanes < 32 && lanes < avg / 8.0) lanes <<= 1;
    D.r_lanes = lanes;
    const double b = 1.1 * L.lmax, a = 0.1 * L.lmax;
    D.theta = static_cast<float>(0.5 * (b + a));
    D.delta = static_cast<float>(0.5 * (b - a));
    D.sigma = static_cast<float>((b + a) / (b - a));
  }
  // coarsest inverse: FP64 Gauss-Jordan on the device, stored FP32
  {
    DevBuf<double> M, colk;
    M.upload(h.coarse_dense, s);
    colk.alloc(std::max<int64_t>(nc, 1));
    const int64_t nn = nc * nc;
    for (int64_t k = 0; k < nc; ++k) {
      k_gj_pivot<<<1, 1024, 0, s>>>(M.p, colk.p, nc, k);
      k_gj_update<<<grid_for(nn, 256), 256, 0, s>>>(M.p, colk.p, nc, k);
    }
    SPX_LAUNCH_CHECK();
    ldc = (nc + 3) / 4 * 4;  // rows of 16-byte vectors
    cinv.alloc(std::max<int64_t>(nc * ldc, 1));
    k_to_float_rows<<<grid_for(nc * ldc, 256), 256, 0, s>>>(M.p, cinv.p, nc, ldc);
    SPX_LAUNCH_CHECK();
    SPX_CUDA(cudaStreamSynchronize(s));
  }
}

int64_t AmgDevice::device_bytes() const {
  int64_t t = cinv.bytes();
  for (int l = 0; l < nlev; ++l) {
    t += A[l].slice_ptr.bytes() + A[l].col.bytes() + P[l].slice_ptr.bytes() + P[l].col.bytes() + rrp[l].bytes() +
         rcol[l].bytes() + val[l].bytes() + pval[l].bytes() + rval[l].bytes() + dinv[l].bytes() + vec[l].bytes();
  }
  return t;
}

// ------------------------------------------------------------------ device phases
namespace {

// 768 threads (80 registers): u1 of the 400x400x2 film / the 64 boxes / the 20x20x5 box 45.5 /
// 34.2 / 6.9 ms per 40 solves; 1024 threads (64 registers, spills) 45.5 / 37.5 / 7.6, 512 threads
// 48.1 / 34.9 / 6.8 (fewer rows in flight)
#ifndef SPX_PCG_BLOCK
#define SPX_PCG_BLOCK 768
#endif
#ifndef SPX_PCG_CTAS_PER_SM
#define SPX_PCG_CTAS_PER_SM 1
#endif
#ifndef SPX_PCG_BLOCK_R
#define SPX_PCG_BLOCK_R 512
#endif
constexpr int PCG_BLOCK = SPX_PCG_BLOCK;          // threads per CTA
// the R-block kernels keep R values per row in registers: fewer threads, more registers each
constexpr int PCG_BLOCK_R = SPX_PCG_BLOCK_R;
constexpr int PCG_CTAS_PER_SM = SPX_PCG_CTAS_PER_SM;  // resident CTAs per SM (all SMs filled)

struct RowRange {
  int64_t gw, nw;  // first warp, warp stride
  int lane;
};

// L2 residency hints.  The cycle's matrices (level 0: ~8 B per nonzero, read five times per
// PCG iteration together with the PCG product) are loaded with an evict_last policy so that
// they stay in L2 across the phases and iterations while vectors, transfer operators and the
// FP64 true-residual values stream past them (those use evict_first where read once).
__device__ __forceinline__ uint64_t l2_policy_keep() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_stream() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ float ld_hint(const float* a, uint64_t pol) {
  float v;
  asm("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ int32_t ld_hint(const int32_t* a, uint64_t pol) {
  int32_t v;
  asm("ld.global.nc.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(v) : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ double ld_hint(const double* a, uint64_t pol) {
  double v;
  asm("ld.global.nc.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ float4 ld_hint4(const float4* a, uint64_t pol) {
  float4 v;
  asm("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(a), "l"(pol));
  return v;
}

// Slice bounds of SELL-32 slice sl (zero width past the last slice); the PCG product phase
// loads the bounds of a warp's next slice while it works on the current one.
__device__ __forceinline__ void slice_bounds(const int64_t* __restrict__ sp, int64_t sl, int64_t ns, int64_t& base,
                                             int& width) {
  if (sl < ns) {
    base = sp[sl];
    width = static_cast<int>((sp[sl + 1] - base) >> 5);
  } else {
    base = 0;
    width = 0;
  }
}

// ---- R identical blocks (a batch of samples of one mesh): the matrix of one block and its
// hierarchy are stored once.  The cycle's level vectors and the PCG work vectors r, p, q hold
// the R blocks interleaved ([row][R]), so the R entries of a column are one vector load (8, 16
// or 32 bytes); the PCG's right-hand side, solution and iterate (b, x, y, bh) keep the
// ensemble's block order ([R][n]).  Each phase reads a matrix slice once.

template <int R> struct VecR;
template <> struct VecR<2> { using T = float2; };
template <> struct VecR<4> { using T = float4; };
template <int R>
__device__ __forceinline__ void load_r(const float* __restrict__ v, int64_t c, float (&g)[R]) {
  if constexpr (R == 8) {
    const float4 a = reinterpret_cast<const float4*>(v + c * 8)[0];
    const float4 b = reinterpret_cast<const float4*>(v + c * 8)[1];
    g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w; g[4] = b.x; g[5] = b.y; g[6] = b.z; g[7] = b.w;
  } else if constexpr (R == 4) {
    const float4 a = reinterpret_cast<const float4*>(v)[c];
    g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w;
  } else if constexpr (R == 2) {
    const float2 a = reinterpret_cast<const float2*>(v)[c];
    g[0] = a.x; g[1] = a.y;
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) g[r] = v[c * R + r];
  }
}

template <int R>
__device__ __forceinline__ void store_r(float* __restrict__ v, int64_t c, const float (&g)[R]) {
  if constexpr (R == 8) {
    reinterpret_cast<float4*>(v + c * 8)[0] = make_float4(g[0], g[1], g[2], g[3]);
    reinterpret_cast<float4*>(v + c * 8)[1] = make_float4(g[4], g[5], g[6], g[7]);
  } else if constexpr (R == 4) {
    reinterpret_cast<float4*>(v)[c] = make_float4(g[0], g[1], g[2], g[3]);
  } else if constexpr (R == 2) {
    reinterpret_cast<float2*>(v)[c] = make_float2(g[0], g[1]);
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) v[c * R + r] = g[r];
  }
}

// R interleaved FP64 entries of row c ([row][R], R even): 16-byte loads and stores
template <int R>
__device__ __forceinline__ void load_r64(const double* __restrict__ v, int64_t c, double (&g)[R]) {
  static_assert(R % 2 == 0, "R even");
  const double2* p = reinterpret_cast<const double2*>(v + c * R);
#pragma unroll
  for (int h = 0; h < R / 2; ++h) {
    const double2 a = p[h];
    g[2 * h] = a.x;
    g[2 * h + 1] = a.y;
  }
}
template <int R>
__device__ __forceinline__ void store_r64(double* __restrict__ v, int64_t c, const double (&g)[R]) {
  double2* p = reinterpret_cast<double2*>(v + c * R);
#pragma unroll
  for (int h = 0; h < R / 2; ++h) p[h] = make_double2(g[2 * h], g[2 * h + 1]);
}

template <int R>
__device__ __forceinline__ void sell_dot_r(const int64_t* __restrict__ sp, const int32_t* __restrict__ col,
                                           const float* __restrict__ val, int64_t sl, int lane,
                                           const float* __restrict__ v, uint64_t pol, float (&t)[R]) {
  constexpr int KB = R >= 8 ? 4 : 8;  // columns in flight per thread
  const int64_t base = sp[sl];
  const int width = static_cast<int>((sp[sl + 1] - base) >> 5);
  const float* vv = val + base + lane;
  const int32_t* cc = col + base + lane;
#pragma unroll
  for (int r = 0; r < R; ++r) t[r] = 0.0f;
  for (int k = 0; k < width; k += KB) {  // the last round predicated
    float w[KB];
    int32_t c[KB];
#pragma unroll
    for (int u = 0; u < KB; ++u) {
      const bool in = k + u < width;
      w[u] = in ? ld_hint(vv + (k + u) * 32, pol) : 0.0f;
      c[u] = in ? ld_hint(cc + (k + u) * 32, pol) : 0;
    }
    float g[KB][R];
#pragma unroll
    for (int u = 0; u < KB; ++u) load_r<R>(v, c[u], g[u]);
#pragma unroll
    for (int u = 0; u < KB; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r) t[r] += w[u] * g[u][r];
  }
}

template <int R>
__device__ void pre_a_r(const AmgLevelDev& L, RowRange rr) {
  const float rho0 = 1.0f / L.sigma, rho1 = 1.0f / (2.0f * L.sigma - rho0);
  for (int64_t sl = rr.gw; sl < L.nslices; sl += rr.nw) {
    const int64_t i = sl * 32 + rr.lane;
    float t[R];
    sell_dot_r<R>(L.sp, L.col, L.val, sl, rr.lane, L.db, l2_policy_keep(), t);
    if (i < L.n) {
      const float di = L.dinv[i];
      float db[R], xo[R], dd[R], ro[R];
      load_r<R>(L.db, i, db);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float d0 = db[r] / L.theta;
        const float r1 = db[r] - di * t[r] / L.theta;
        const float d1 = rho1 * rho0 * d0 + (2.0f * rho1 / L.delta) * r1;
        xo[r] = d0 + d1;
        dd[r] = d1;
        ro[r] = r1;
      }
      store_r<R>(L.x, i, xo);
      store_r<R>(L.d, i, dd);
      store_r<R>(L.r, i, ro);
    }
  }
}

template <int R>
__device__ void pre_b_r(const AmgLevelDev& L, RowRange rr) {
  for (int64_t sl = rr.gw; sl < L.nslices; sl += rr.nw) {
    const int64_t i = sl * 32 + rr.lane;
    float t[R];
    sell_dot_r<R>(L.sp, L.col, L.val, sl, rr.lane, L.d, l2_policy_keep(), t);
    if (i < L.n) {
      const float di = L.dinv[i];
      float rv[R];
      load_r<R>(L.r, i, rv);
#pragma unroll
      for (int r = 0; r < R; ++r) rv[r] = (rv[r] - di * t[r]) / di;
      store_r<R>(L.r, i, rv);
    }
  }
}

template <int R>
__device__ void restrict_to_r(const AmgLevelDev& L, const AmgLevelDev& C, RowRange rr) {
  const int G = L.r_lanes;
  const int gl = rr.lane & (G - 1);
  const int64_t rows_per_warp = 32 / G;
  const int64_t first = rr.gw * rows_per_warp + rr.lane / G, stride = rr.nw * rows_per_warp;
  const int64_t nrows_pad = (C.n + rows_per_warp - 1) / rows_per_warp * rows_per_warp;
  for (int64_t a = first - rr.lane / G; a < nrows_pad; a += stride) {  // uniform per warp
    const int64_t row = a + rr.lane / G;
    float t[R];
#pragma unroll
    for (int r = 0; r < R; ++r) t[r] = 0.0f;
    if (row < C.n) {
      const int64_t k1 = L.r_rp[row + 1];
      int64_t k = L.r_rp[row] + gl;
      for (; k + G < k1; k += 2 * G) {  // two gathers in flight per lane
        const float w0 = L.r_val[k], w1 = L.r_val[k + G];
        const int32_t c0 = L.r_col[k], c1 = L.r_col[k + G];
        float g0[R], g1[R];
        load_r<R>(L.r, c0, g0);
        load_r<R>(L.r, c1, g1);
#pragma unroll
        for (int r = 0; r < R; ++r) t[r] += w0 * g0[r] + w1 * g1[r];
      }
      for (; k < k1; k += G) {
        const float w = L.r_val[k];
        float g[R];
        load_r<R>(L.r, L.r_col[k], g);
#pragma unroll
        for (int r = 0; r < R; ++r) t[r] += w * g[r];
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
      for (int o = G >> 1; o > 0; o >>= 1) t[r] += __shfl_xor_sync(0xffffffffu, t[r], o);
    if (row < C.n && gl == 0) {
      const float dc = C.dinv[row];
      float dbv[R];
#pragma unroll
      for (int r = 0; r < R; ++r) dbv[r] = dc * t[r];
      store_r<R>(C.b, row, t);
      store_r<R>(C.db, row, dbv);
    }
  }
}

template <int R>
__device__ void prolong_from_r(const AmgLevelDev& L, const AmgLevelDev& C, RowRange rr) {
  for (int64_t sl = rr.gw; sl < L.p_nslices; sl += rr.nw) {
    const int64_t i = sl * 32 + rr.lane;
    float t[R];
    sell_dot_r<R>(L.p_sp, L.p_col, L.p_val, sl, rr.lane, C.x, l2_policy_stream(), t);
    if (i < L.n) {
      float xv[R];
      load_r<R>(L.x, i, xv);
#pragma unroll
      for (int r = 0; r < R; ++r) xv[r] += t[r];
      store_r<R>(L.x, i, xv);
    }
  }
}

template <int R>
__device__ void post_c_r(const AmgLevelDev& L, RowRange rr) {
  for (int64_t sl = rr.gw; sl < L.nslices; sl += rr.nw) {
    const int64_t i = sl * 32 + rr.lane;
    float t[R];
    sell_dot_r<R>(L.sp, L.col, L.val, sl, rr.lane, L.x, l2_policy_keep(), t);
    if (i < L.n) {
      const float di = L.dinv[i];
      float db[R], xv[R], x2[R], dd[R], ro[R];
      load_r<R>(L.db, i, db);
      load_r<R>(L.x, i, xv);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float r0 = db[r] - di * t[r];
        const float d0 = r0 / L.theta;
        x2[r] = xv[r] + d0;
        dd[r] = d0;
        ro[r] = r0;
      }
      store_r<R>(L.x2, i, x2);
      store_r<R>(L.d, i, dd);
      store_r<R>(L.r, i, ro);
    }
  }
}

// on the top level also the partial dots (r64, u), (d, u) over all R blocks; r64 is the
// interleaved PCG residual, diag the (replicated) diagonal
template <int R>
__device__ void post_d_r(const AmgLevelDev& L, RowRange rr, const double* __restrict__ r64,
                         const double* __restrict__ diag, double& rz, double& wz, bool top) {
  const float rho0 = 1.0f / L.sigma, rho1 = 1.0f / (2.0f * L.sigma - rho0);
  for (int64_t sl = rr.gw; sl < L.nslices; sl += rr.nw) {
    const int64_t i = sl * 32 + rr.lane;
    float t[R];
    sell_dot_r<R>(L.sp, L.col, L.val, sl, rr.lane, L.d, l2_policy_keep(), t);
    if (i < L.n) {
      const float di = L.dinv[i];
      const double dg = top ? diag[i] : 0.0;
      float rv[R], dv[R], x2[R], zo[R];
      load_r<R>(L.r, i, rv);
      load_r<R>(L.d, i, dv);
      load_r<R>(L.x2, i, x2);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float r1 = rv[r] - di * t[r];
        const float d1 = rho1 * rho0 * dv[r] + (2.0f * rho1 / L.delta) * r1;
        const float z = x2[r] + d1;
        zo[r] = z;
        if (top) {
          rz += r64[i * R + r] * static_cast<double>(z);
          wz += dg * static_cast<double>(z);
        }
      }
      store_r<R>(L.x, i, zo);
    }
  }
}

// the right-hand sides of the dense coarsest level, transposed to [R][nc], for k_pcg_amg_r's
// coarse phase (dynamic shared memory of nc x R floats)
extern __shared__ float pcg_coarse_smem[];

// dense coarsest level for R blocks (interleaved vectors): the CTA stages the R right-hand
// sides in shared memory ([R][nc], one coalesced pass), then a warp per row of the inverse
// reads the row once (L2 evict_last policy, coalesced) against all R of them
template <int R>
__device__ void coarse_solve_r(const AmgLevelDev& L, const float* __restrict__ cinv, int64_t nc, int64_t ldc,
                               RowRange rr) {
  float* sb = pcg_coarse_smem;
  for (int64_t e = threadIdx.x; e < nc * R; e += blockDim.x) {
    const int64_t j = e / R;
    sb[(e - j * R) * nc + j] = L.b[e];
  }
  __syncthreads();
  const uint64_t pol = l2_policy_keep();  // the inverse stays in L2 across iterations
  for (int64_t i = rr.gw; i < nc; i += rr.nw) {
    const float* row = cinv + i * ldc;
    float s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] = 0.0f;
#pragma unroll 4
    for (int64_t j = rr.lane; j < nc; j += 32) {
      const float c = ld_hint(row + j, pol);
#pragma unroll
      for (int r = 0; r < R; ++r) s[r] += c * sb[r * nc + j];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      for (int o = 16; o > 0; o >>= 1) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
      if (rr.lane == 0) L.x[i * R + r] = s[r];
    }
  }
}

template <class TV>
struct PcgParams {
  int64_t n, nslices;
  const int64_t* sp;
  const int32_t* col;
  const double* a64;   // FP64 values (true residual)
  const float* a32;    // FP32 values (difference-form SpMV)
  const double* rsum;  // row sums of the matrix
  const double* diag;
  const TV* b;
  TV* x;
  double *bh, *y, *r, *p, *q;
  double* part;
  unsigned int* bar;
  int* err;
  int* iters;
  double* resid;
  unsigned long long* iters_acc;
  double* res_acc;
  double rtol, atol, ww;
  int maxit, max_outer, warm, project;
  int bh_given;  // bh already holds the projected right-hand side (FP64)
  int nlev;
  const float* cinv;
  int64_t nc, ldc;
  int reps;  // identical blocks: vectors hold reps x n entries, the matrix n rows
  int timing;  // phase timing marks on (spx_debug_pcg_timing)
  AmgLevelDev L[AMG_MAX_LEVELS];
  AmgResident R[AMG_MAX_LEVELS];
};

#define PCG_ROWS_BEGIN                                              \
  for (int64_t sl = gw; sl < P.nslices; sl += nw) {                 \
    const int64_t row = sl * 32 + lane;                             \
    const int64_t base = P.sp[sl];                                  \
    const int width = static_cast<int>((P.sp[sl + 1] - base) >> 5); \
    (void)base; (void)width;                                        \
    if (row < n) {
#define PCG_ROWS_END \
  }                  \
  }
// SpMV phases: the bounds of the warp's next slice are loaded while it works on this one
#define PCG_SLICES_BEGIN                                     \
  {                                                          \
    int64_t base, nbase_;                                    \
    int width, nwidth_;                                      \
    slice_bounds(P.sp, gw, P.nslices, base, width);          \
    for (int64_t sl = gw; sl < P.nslices; sl += nw) {        \
      slice_bounds(P.sp, sl + nw, P.nslices, nbase_, nwidth_); \
      const int64_t row = sl * 32 + lane;                    \
      if (row < n) {
#define PCG_SLICES_END \
  }                    \
  base = nbase_;       \
  width = nwidth_;     \
  }                    \
  }

// Phase timing of k_pcg_amg and k_pcg_amg_r (switched on by spx_debug_pcg_timing): CTA 0 adds the globaltimer interval
// since its previous mark to the slot of the phase that just ended (the phase's slowest CTA
// plus the barrier); read and cleared by pcg_phase_times.  Slots: V-cycle phases in order
// (3 per level down, the coarse solve, 3 per level up), 28 the PCG product, 29 the update,
// 30 the true residual.
__device__ unsigned long long g_pcg_phase_ns[32];
__device__ unsigned long long g_pcg_phase_n[32];
__device__ __forceinline__ void pcg_mark(unsigned long long& t_prev, int slot, int on) {
  if (on && blockIdx.x == 0 && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t_prev != 0ull && slot >= 0 && slot < 32) {
      g_pcg_phase_ns[slot] += t - t_prev;
      g_pcg_phase_n[slot] += 1ull;
    }
    t_prev = t;
  }
}

// ---- one system (k_pcg_amg): CTA-owned blocks of slices, kept in shared memory
extern __shared__ __align__(16) int32_t pcg_words[];
constexpr int PCG_DYN_MAX = 220 * 1024;  // dynamic shared memory; the rest is for static data and L1

// this CTA's block of one level: slices [s0, s0 + cnt), the first nres of them resident
struct LvlBlock {
  int64_t s0;
  int64_t base, pbase;  // first entries of the block's rows of A and P in global memory
  int64_t r0, rbase;  // coarse rows [r0, r0 + rcnt) of the restriction, their first entry
  int32_t cnt, nres, rcnt;
};
struct PcgShared {
  LvlBlock blk[AMG_MAX_LEVELS];
  double red[64], tot[2];
  int ok;
};

// bounds of slice k of the block, relative to its first entry
__device__ __forceinline__ void block_bounds(const AmgLevelDev& L, const AmgResident& R, const LvlBlock& B, int k,
                                             int64_t& o, int& width) {
  if (R.off >= 0) {
    const int32_t a = pcg_words[R.off + k], e = pcg_words[R.off + k + 1];
    o = a;
    width = (e - a) >> 5;
  } else {
    const int64_t a = L.sp[B.s0 + k];
    o = a - B.base;
    width = static_cast<int>((L.sp[B.s0 + k + 1] - a) >> 5);
  }
}

// sum_k w_k f(v[c_k]) over the entries of one row: eight gathers in flight; entries from shared
// memory (resident slice) or through L2.  f is applied to the gathered value.
template <class TA, class F>
__device__ __forceinline__ TA block_dot(const AmgLevelDev& L, const AmgResident& R, const LvlBlock& B, int k, int lane,
                                        const float* v, F f) {
  int64_t o;
  int width;
  block_bounds(L, R, B, k, o, width);
  TA a0 = TA(0), a1 = TA(0);
  if (k < B.nres) {
    const int wv = R.val + static_cast<int>(o) + lane, wc = R.col + static_cast<int>(o) + lane;
    for (int j = 0; j < width; j += 8) {
      float g[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) g[u] = j + u < width ? v[pcg_words[wc + (j + u) * 32]] : 0.0f;
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        if (j + u < width) a0 += static_cast<TA>(__int_as_float(pcg_words[wv + (j + u) * 32])) * f(g[u]);
        if (j + u + 1 < width) a1 += static_cast<TA>(__int_as_float(pcg_words[wv + (j + u + 1) * 32])) * f(g[u + 1]);
      }
    }
  } else {
    const uint64_t pol = l2_policy_keep();
    const float* gv = L.val + B.base + o + lane;
    const int32_t* gc = L.col + B.base + o + lane;
    for (int j = 0; j < width; j += 8) {
      int32_t c[8];
      float w[8], g[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const bool in = j + u < width;
        c[u] = in ? ld_hint(gc + (j + u) * 32, pol) : 0;
        w[u] = in ? ld_hint(gv + (j + u) * 32, pol) : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) g[u] = j + u < width ? v[c[u]] : 0.0f;
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        if (j + u < width) a0 += static_cast<TA>(w[u]) * f(g[u]);
        if (j + u + 1 < width) a1 += static_cast<TA>(w[u + 1]) * f(g[u + 1]);
      }
    }
  }
  return a0 + a1;
}
__device__ __forceinline__ float block_dot(const AmgLevelDev& L, const AmgResident& R, const LvlBlock& B, int k,
                                           int lane, const float* v) {
  return block_dot<float>(L, R, B, k, lane, v, [](float g) { return g; });
}

// rows of this CTA's block of a level; the body sees k (slice of the block) and i (row)
#define BLOCK_ROWS_BEGIN(B, nrows)                                              \
  for (int k = threadIdx.x >> 5; k < (B).cnt; k += blockDim.x >> 5) {           \
    const int lane = threadIdx.x & 31;                                          \
    const int64_t i = ((B).s0 + k) * 32 + lane;                                 \
    if (i < (nrows)) {
#define BLOCK_ROWS_END \
  }                    \
  }

// pre-smoothing from x = 0, Chebyshev steps 1 and 2 (one SpMV: A d0, d0 = D^-1 b / theta)
__device__ __forceinline__ void pre_a(const AmgLevelDev& L, const AmgResident& R, const LvlBlock& B) {
  const float rho0 = 1.0f / L.sigma, rho1 = 1.0f / (2.0f * L.sigma - rho0);
  const float it = 1.0f / L.theta, c0 = rho1 * rho0, c1 = 2.0f * rho1 / L.delta;
  BLOCK_ROWS_BEGIN(B, L.n)
    const float di = L.dinv[i], db = L.db[i];
    const float t = block_dot(L, R, B, k, lane, L.db);
    const float d0 = db * it;
    const float r1 = db - di * t * it;
    const float d1 = c0 * d0 + c1 * r1;
    L.x[i] = d0 + d1;
    L.d[i] = d1;
    L.r[i] = r1;
  BLOCK_ROWS_END
}

// residual b - A x after pre-smoothing (A d1), stored in r
__device__ __forceinline__ void pre_b(const AmgLevelDev& L, const AmgResident& R, const LvlBlock& B) {
  BLOCK_ROWS_BEGIN(B, L.n)
    const float di = L.dinv[i], r = L.r[i];
    const float t = block_dot(L, R, B, k, lane, L.d);
    L.r[i] = r / di - t;
  BLOCK_ROWS_END
}

// b_c = R r (CSR rows, `r_lanes` lanes per row), db_c = D_c^-1 b_c; each CTA takes a contiguous
// block of the coarse rows, whose bounds it keeps in shared memory
__device__ __forceinline__ void restrict_to(const AmgLevelDev& L, const AmgResident& R, const LvlBlock& B,
                                            const AmgLevelDev& C) {
  const int lane = threadIdx.x & 31, G = L.r_lanes, gl = lane & (G - 1), rpw = 32 / G;
  for (int a = (threadIdx.x >> 5) * rpw; a < B.rcnt; a += (blockDim.x >> 5) * rpw) {  // uniform per warp
    const int q = a + lane / G;
    const int64_t row = B.r0 + q;
    float t = 0.0f, di = 0.0f;
    if (q < B.rcnt) {
      int64_t k, k1;
      if (R.off >= 0) {
        k = B.rbase + pcg_words[R.roff + q] + gl;
        k1 = B.rbase + pcg_words[R.roff + q + 1];
      } else {
        k = L.r_rp[row] + gl;
        k1 = L.r_rp[row + 1];
      }
      di = C.dinv[row];
      for (; k < k1; k += 8 * G) {  // eight gathers in flight per lane
        int32_t c[8];
        float w[8], g[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const bool in = k + u * G < k1;
          c[u] = in ? L.r_col[k + u * G] : 0;
          w[u] = in ? L.r_val[k + u * G] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) g[u] = k + u * G < k1 ? L.r[c[u]] : 0.0f;
#pragma unroll
        for (int u = 0; u < 8; ++u) t += w[u] * g[u];
      }
    }
    for (int o = G >> 1; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (q < B.rcnt && gl == 0) {
      C.b[row] = t;
      C.db[row] = di * t;
    }
  }
}

// x += P x_c; P has the rows of L and so its slices (L's block)
__device__ __forceinline__ void prolong_from(const AmgLevelDev& L, const AmgResident& R, const AmgLevelDev& C,
                                             const LvlBlock& B) {
  BLOCK_ROWS_BEGIN(B, L.n)
    int64_t base;
    int width;
    if (R.off >= 0) {
      const int32_t o = pcg_words[R.poff + k];
      base = B.pbase + o;
      width = (pcg_words[R.poff + k + 1] - o) >> 5;
    } else {
      base = L.p_sp[B.s0 + k];
      width = static_cast<int>((L.p_sp[B.s0 + k + 1] - base) >> 5);
    }
    const float xi = L.x[i];
    const float* pv = L.p_val + base + lane;
    const int32_t* pc = L.p_col + base + lane;
    float t = 0.0f;
    for (int j = 0; j < width; j += 4) {
      int32_t c[4];
      float w[4], g[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool in = j + u < width;
        c[u] = in ? pc[(j + u) * 32] : 0;
        w[u] = in ? pv[(j + u) * 32] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) g[u] = j + u < width ? C.x[c[u]] : 0.0f;
#pragma unroll
      for (int u = 0; u < 4; ++u) t += w[u] * g[u];
    }
    L.x[i] = xi + t;
  BLOCK_ROWS_END
}

// post-smoothing from x, Chebyshev step 1 (r0 = D^-1 (b - A x), x2 = x + r0 / theta)
__device__ __forceinline__ void post_c(const AmgLevelDev& L, const AmgResident& R, const LvlBlock& B) {
  const float it = 1.0f / L.theta;
  BLOCK_ROWS_BEGIN(B, L.n)
    const float di = L.dinv[i], db = L.db[i], x = L.x[i];
    const float t = block_dot(L, R, B, k, lane, L.x);
    const float r0 = db - di * t;
    L.x2[i] = x + r0 * it;
    L.r[i] = r0;
  BLOCK_ROWS_END
}

// post-smoothing step 2 (d0 = r0 / theta); on the top level also the partial dots (r64, u) and
// (d, u) of the PCG
template <bool TOP>
__device__ __forceinline__ void post_d(const AmgLevelDev& L, const AmgResident& R, const LvlBlock& B, const double* r64,
                                       const double* diag, double& rz, double& wz) {
  const float rho0 = 1.0f / L.sigma, rho1 = 1.0f / (2.0f * L.sigma - rho0);
  const float it = 1.0f / L.theta, c0 = rho1 * rho0 * it, c1 = 2.0f * rho1 / L.delta;
  BLOCK_ROWS_BEGIN(B, L.n)
    const float di = L.dinv[i], r0 = L.r[i], x2 = L.x2[i];
    const double rd = TOP ? r64[i] : 0.0, dg = TOP ? diag[i] : 0.0;
    const float t = block_dot(L, R, B, k, lane, L.r) * it;
    const float r1 = r0 - di * t;
    const float z = x2 + (c0 * r0 + c1 * r1);
    L.x[i] = z;
    if (TOP) {
      rz += rd * static_cast<double>(z);
      wz += dg * static_cast<double>(z);
    }
  BLOCK_ROWS_END
}

// x = C^-1 b on the dense coarsest level: each CTA takes a contiguous block of rows, its warps
// split evenly over them (several warps to a row on the few rows of a CTA, their sums joined in
// shared memory); 16-byte loads of the zero-padded rows (ld = nc rounded up to 4; b is read up
// to ld, inside the level's vectors), nine of a lane in flight.
__device__ __forceinline__ void coarse_solve(const AmgLevelDev& L, const float* __restrict__ cinv, int64_t nc,
                                             int64_t ldc, double* red) {
  const int nv = static_cast<int>(ldc / 4), warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = static_cast<int>(nc * blockIdx.x / gridDim.x), r1 = static_cast<int>(nc * (blockIdx.x + 1) / gridDim.x);
  const uint64_t pol = l2_policy_keep();  // the inverse stays in L2 across iterations
  const float4* b4 = reinterpret_cast<const float4*>(L.b);
  float* fr = reinterpret_cast<float*>(red);
  int wpr = 1;  // warps per row
  while (wpr * 2 * (r1 - r0) <= warps && wpr < 32) wpr *= 2;
  const int rows = warps / wpr, part = warp & (wpr - 1);
  for (int a = r0; a < r1; a += rows) {  // uniform per CTA
    const int i = a + warp / wpr;
    float s = 0.0f;
    if (i < r1) {
      const float4* row = reinterpret_cast<const float4*>(cinv + static_cast<int64_t>(i) * ldc);
#pragma unroll 9
      for (int j = part * 32 + lane; j < nv; j += 32 * wpr) {
        const float4 c = ld_hint4(row + j, pol);
        const float4 b = b4[j];
        s += c.x * b.x + c.y * b.y + c.z * b.z + c.w * b.w;
      }
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (wpr == 1) {
      if (lane == 0 && i < r1) L.x[i] = s;
    } else {
      if (lane == 0) fr[warp] = s;
      __syncthreads();
      if (part == 0 && lane == 0 && i < r1) {
        for (int q = 1; q < wpr; ++q) s += fr[warp + q];
        L.x[i] = s;
      }
      __syncthreads();
    }
  }
}

// Grid barrier with two sums: every CTA's partials of a and b are written before its arrival and
// added up, in the same order in every CTA, by the waiting warp before it releases its CTA.
// `flip` alternates the two slots of the partials: a CTA writes a slot again only after the
// barrier that follows every CTA's last read of it.  Bounded wait as in grid_barrier.
template <class TV>
__device__ __forceinline__ bool sync_sum(const PcgParams<TV>& P, PcgShared& S, int& flip, double& a, double& b) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nb = gridDim.x;
  a = warp_sum(a);
  b = warp_sum(b);
  if (lane == 0) {
    S.red[2 * wid] = a;
    S.red[2 * wid + 1] = b;
  }
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    double u = warp_sum(lane < nw ? S.red[2 * lane] : 0.0);
    double v = warp_sum(lane < nw ? S.red[2 * lane + 1] : 0.0);
    double* part = P.part + static_cast<int64_t>(flip) * 2 * nb;
    int ok = 1;
    if (lane == 0) {
      part[2 * blockIdx.x] = u;
      part[2 * blockIdx.x + 1] = v;
      ok = grid_arrive_wait(P.bar, nb, P.err) ? 1 : 0;
      S.ok = ok;
    }
    __syncwarp();
    u = v = 0.0;
    for (int c = lane; c < nb; c += 32) {
      const double2 q = __ldcg(reinterpret_cast<const double2*>(part) + c);
      u += q.x;
      v += q.y;
    }
    u = warp_sum(u);
    v = warp_sum(v);
    if (lane == 0) {
      S.tot[0] = u;
      S.tot[1] = v;
    }
  }
  flip ^= 1;
  __syncthreads();
  a = S.tot[0];
  b = S.tot[1];
  return S.ok != 0;
}

// End of one run of PCG iterations: a little below the target, so that the true residual confirms
// it, or 13 digits below the run's first residual: what is left of the recurrence is then near
// its rounding error (a warm start 10^3 times worse than zero, with rtol 1e-13, never reached
// the target within one run), and the next run starts from the true residual.
__device__ __forceinline__ bool pcg_stop(double rr, double rr_start, double tol2) {
  return rr <= 0.25 * tol2 || rr <= 1e-26 * rr_start;
}

// u = V(r): L[0].db holds D^-1 r (FP32) on entry, L[0].x holds u on exit; rz, wz: (r, u), (d, u)
// over the grid.  nlev >= 2.
template <class TV>
__device__ __forceinline__ bool vcycle(const PcgParams<TV>& P, PcgShared& S, int& flip, double& rz, double& wz,
                                       unsigned long long& tm) {
  const unsigned nb = gridDim.x;
  unsigned int* cnt = P.bar;
  const int NL = P.nlev;
  int ph = 0;
  for (int l = 0; l + 1 < NL; ++l) {
    const AmgLevelDev& L = P.L[l];
    pre_a(L, P.R[l], S.blk[l]);
    if (!grid_barrier(cnt, nullptr, nb, P.err)) return false;
    pcg_mark(tm, ph++, P.timing);
    pre_b(L, P.R[l], S.blk[l]);
    if (!grid_barrier(cnt, nullptr, nb, P.err)) return false;
    pcg_mark(tm, ph++, P.timing);
    restrict_to(L, P.R[l], S.blk[l], P.L[l + 1]);
    if (!grid_barrier(cnt, nullptr, nb, P.err)) return false;
    pcg_mark(tm, ph++, P.timing);
  }
  coarse_solve(P.L[NL - 1], P.cinv, P.nc, P.ldc, S.red);
  if (!grid_barrier(cnt, nullptr, nb, P.err)) return false;
  pcg_mark(tm, ph++, P.timing);
  rz = wz = 0.0;
  for (int l = NL - 2; l >= 0; --l) {
    const AmgLevelDev& L = P.L[l];
    prolong_from(L, P.R[l], P.L[l + 1], S.blk[l]);
    if (!grid_barrier(cnt, nullptr, nb, P.err)) return false;
    pcg_mark(tm, ph++, P.timing);
    post_c(L, P.R[l], S.blk[l]);
    if (!grid_barrier(cnt, nullptr, nb, P.err)) return false;
    pcg_mark(tm, ph++, P.timing);
    if (l == 0) {
      post_d<true>(L, P.R[l], S.blk[l], P.r, P.diag, rz, wz);
      if (!sync_sum(P, S, flip, rz, wz)) return false;
    } else {
      post_d<false>(L, P.R[l], S.blk[l], nullptr, nullptr, rz, wz);
      if (!grid_barrier(cnt, nullptr, nb, P.err)) return false;
    }
    pcg_mark(tm, ph++, P.timing);
  }
  return true;
}

template <class TV>
__global__ void __launch_bounds__(PCG_BLOCK, PCG_CTAS_PER_SM) k_pcg_amg(const __grid_constant__ PcgParams<TV> P) {
  unsigned long long tm = 0ull;
  __shared__ PcgShared S;
  int flip = 0;
  const int64_t n = P.n;
  // this CTA's blocks: bounds, how much of each is resident, the resident entries
  for (int l = threadIdx.x; l + 1 < P.nlev; l += blockDim.x) {
    LvlBlock B;
    B.s0 = P.L[l].nslices * blockIdx.x / gridDim.x;
    B.cnt = static_cast<int32_t>(P.L[l].nslices * (blockIdx.x + 1) / gridDim.x - B.s0);
    B.base = P.L[l].sp[B.s0];
    B.pbase = P.L[l].p_sp[B.s0];
    B.nres = 0;
    const int64_t ncr = P.L[l + 1].n;
    B.r0 = ncr * blockIdx.x / gridDim.x;
    B.rcnt = static_cast<int32_t>(ncr * (blockIdx.x + 1) / gridDim.x - B.r0);
    B.rbase = P.L[l].r_rp[B.r0];
    S.blk[l] = B;
  }
  __syncthreads();
  for (int l = 0; l + 1 < P.nlev; ++l) {
    const LvlBlock& B = S.blk[l];
    if (P.R[l].off >= 0)
      for (int k = threadIdx.x; k <= B.cnt; k += blockDim.x) {
        pcg_words[P.R[l].off + k] = static_cast<int32_t>(P.L[l].sp[B.s0 + k] - B.base);
        pcg_words[P.R[l].poff + k] = static_cast<int32_t>(P.L[l].p_sp[B.s0 + k] - B.pbase);
      }
    if (P.R[l].off >= 0)
      for (int k = threadIdx.x; k <= B.rcnt; k += blockDim.x)
        pcg_words[P.R[l].roff + k] = static_cast<int32_t>(P.L[l].r_rp[B.r0 + k] - B.rbase);
  }
  __syncthreads();
  if (threadIdx.x < P.nlev - 1 && P.R[threadIdx.x].off >= 0) {  // last slice bound within the capacity
    const int l = threadIdx.x;
    int lo = 0, hi = S.blk[l].cnt;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (pcg_words[P.R[l].off + mid] <= P.R[l].cap) lo = mid; else hi = mid - 1;
    }
    S.blk[l].nres = lo;
  }
  __syncthreads();
  for (int l = 0; l + 1 < P.nlev; ++l) {
    const LvlBlock& B = S.blk[l];
    if (B.nres == 0) continue;
    const int m4 = pcg_words[P.R[l].off + B.nres] / 4;  // whole 32-entry columns
    const float4* gv = reinterpret_cast<const float4*>(P.L[l].val + B.base);
    const int4* gc = reinterpret_cast<const int4*>(P.L[l].col + B.base);
    float4* sv = reinterpret_cast<float4*>(pcg_words + P.R[l].val);
    int4* sc = reinterpret_cast<int4*>(pcg_words + P.R[l].col);
    for (int k = threadIdx.x; k < m4; k += blockDim.x) {
      sv[k] = gv[k];
      sc[k] = gc[k];
    }
  }
  __syncthreads();
  const LvlBlock B0 = S.blk[0];
  const AmgLevelDev& L0 = P.L[0];
  double meanb = 0.0, dummy = 0.0;
  if (P.project && !P.bh_given) {
    double part = 0.0;
    BLOCK_ROWS_BEGIN(B0, n) part += static_cast<double>(P.b[i]);
    BLOCK_ROWS_END
    if (!sync_sum(P, S, flip, part, dummy)) return;
    meanb = part / static_cast<double>(n);
  }
  double bb = 0.0;
  BLOCK_ROWS_BEGIN(B0, n)
    double bv;
    if (P.bh_given) {
      bv = P.bh[i];
    } else {
      bv = static_cast<double>(P.b[i]) - meanb;
      P.bh[i] = bv;
    }
    if (!P.warm) P.y[i] = 0.0;
    bb += bv * bv;
  BLOCK_ROWS_END
  dummy = 0.0;
  if (!sync_sum(P, S, flip, bb, dummy)) return;
  if (P.warm && !(bb > 0.0)) {  // b = 0: the solution is 0
    BLOCK_ROWS_BEGIN(B0, n) P.y[i] = 0.0;
    BLOCK_ROWS_END
    if (!grid_barrier(P.bar, nullptr, gridDim.x, P.err)) return;
  }
  const double tol2 = fmax(P.rtol * P.rtol * bb, P.atol * P.atol);
  int total = 0, outers = 0;
  double rr = 0.0, rr0 = -1.0;
  for (int outer = 0; outer < P.max_outer; ++outer) {
    ++outers;
    // true residual r = bh - A y (FP64), its norm, D^-1 r -> level-0 right-hand side
    {
      double rh = 0.0;
      const uint64_t pst = l2_policy_stream();
      BLOCK_ROWS_BEGIN(B0, n)
        int64_t o;
        int width;
        block_bounds(L0, P.R[0], B0, k, o, width);
        const double bv = P.bh[i];
        const float di = L0.dinv[i];
        const double* gv = P.a64 + B0.base + o + lane;
        const int32_t* gc = P.col + B0.base + o + lane;
        const bool res = k < B0.nres;
        const int wc = P.R[0].col + static_cast<int>(res ? o : 0) + lane;
        double acc = 0.0, acc2 = 0.0;
        for (int j = 0; j < width; j += 4) {
          double w[4], g[4];
          int32_t c[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const bool in = j + u < width;
            c[u] = in ? (res ? pcg_words[wc + (j + u) * 32] : gc[(j + u) * 32]) : 0;
            w[u] = in ? ld_hint(gv + (j + u) * 32, pst) : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) g[u] = j + u < width ? P.y[c[u]] : 0.0;
#pragma unroll
          for (int u = 0; u < 4; u += 2) {
            acc += w[u] * g[u];
            acc2 += w[u + 1] * g[u + 1];
          }
        }
        const double r = bv - (acc + acc2);
        P.r[i] = r;
        L0.db[i] = di * static_cast<float>(r);
        rh += r * r;
      BLOCK_ROWS_END
      dummy = 0.0;
      if (!sync_sum(P, S, flip, rh, dummy)) return;
      pcg_mark(tm, 30, P.timing);
      rr = rh;
    }
    if (rr0 < 0.0) rr0 = rr;
    if (rr <= tol2 || total >= P.maxit) break;
    const double rr_start = rr;
    double rz_old = 1.0;
    for (int it = 0;; ++it) {
      double rz, wz;
      if (!vcycle(P, S, flip, rz, wz, tm)) return;
      const double c = P.project && P.ww > 0.0 ? wz / P.ww : 0.0;
      const double beta = it == 0 ? 0.0 : rz / rz_old;
      const float* u0 = L0.x;  // u from the level-0 cycle
      double pq = 0.0;
      BLOCK_ROWS_BEGIN(B0, n)
        const double ui = static_cast<double>(u0[i]), rsi = P.rsum[i];
        const double pold = it == 0 ? 0.0 : P.p[i], qold = it == 0 ? 0.0 : P.q[i];
        const double acc = block_dot<double>(L0, P.R[0], B0, k, lane, u0,
                                             [ui](float g) { return static_cast<double>(g) - ui; });
        const double pv = (ui - c) + (it == 0 ? 0.0 : beta * pold);
        const double qv = (acc + rsi * ui) + (it == 0 ? 0.0 : beta * qold);
        P.p[i] = pv;
        P.q[i] = qv;
        pq += pv * qv;
      BLOCK_ROWS_END
      dummy = 0.0;
      if (!sync_sum(P, S, flip, pq, dummy)) return;
      pcg_mark(tm, 28, P.timing);
      if (!(pq > 0.0) || !(rz > 0.0)) break;
      const double alpha = rz / pq;
      double rh = 0.0;
      BLOCK_ROWS_BEGIN(B0, n)
        const double pv = P.p[i], qv = P.q[i], yv = P.y[i], rv = P.r[i];
        const float di = L0.dinv[i];
        P.y[i] = yv + alpha * pv;
        const double r = rv - alpha * qv;
        P.r[i] = r;
        L0.db[i] = di * static_cast<float>(r);
        rh += r * r;
      BLOCK_ROWS_END
      dummy = 0.0;
      if (!sync_sum(P, S, flip, rh, dummy)) return;
      pcg_mark(tm, 29, P.timing);
      rr = rh;
      ++total;
      rz_old = rz;
      if (pcg_stop(rr, rr_start, tol2) || total >= P.maxit) break;
    }
  }
  double mx = 0.0;
  if (P.project) {
    double sx = 0.0;
    BLOCK_ROWS_BEGIN(B0, n) sx += P.y[i];
    BLOCK_ROWS_END
    dummy = 0.0;
    if (!sync_sum(P, S, flip, sx, dummy)) return;
    mx = sx / static_cast<double>(n);
  }
  BLOCK_ROWS_BEGIN(B0, n)
    const double xv = P.y[i] - mx;
    P.x[i] = static_cast<TV>(xv);
    P.y[i] = xv;
  BLOCK_ROWS_END
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *P.iters = total;
    *P.resid = bb > 0.0 ? sqrt(rr / bb) : 0.0;
    atomicAdd(P.iters_acc, (unsigned long long)total);
    atomicAdd(P.iters_acc + 1, (unsigned long long)outers);
    atomicAdd(P.iters_acc + 2, 1ull);
    if (bb > 0.0) {
      atomicAdd(P.res_acc, sqrt(fmax(rr0, 0.0) / bb));
      atomicAdd(P.res_acc + 1, sqrt(rr / bb));
    }
  }
}

// the V-cycle of k_pcg_amg for R identical blocks (same phases and barriers)
template <class TV, int R>
__device__ bool vcycle_r(const PcgParams<TV>& P, int slot, double* sh, unsigned long long& tm) {
  const unsigned nb = gridDim.x;
  unsigned int* cnt = P.bar;
  unsigned int* gen = P.bar + 1;
  const RowRange rr{static_cast<int64_t>((blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5),
                    static_cast<int64_t>((gridDim.x * static_cast<int64_t>(blockDim.x)) >> 5),
                    static_cast<int>(threadIdx.x & 31)};
  const int NL = P.nlev;
  int ph = 0;
  for (int l = 0; l + 1 < NL; ++l) {
    const AmgLevelDev& L = P.L[l];
    pre_a_r<R>(L, rr);
    if (!grid_barrier(cnt, gen, nb, P.err)) return false;
    pcg_mark(tm, ph++, P.timing);
    pre_b_r<R>(L, rr);
    if (!grid_barrier(cnt, gen, nb, P.err)) return false;
    pcg_mark(tm, ph++, P.timing);
    restrict_to_r<R>(L, P.L[l + 1], rr);
    if (!grid_barrier(cnt, gen, nb, P.err)) return false;
    pcg_mark(tm, ph++, P.timing);
  }
  coarse_solve_r<R>(P.L[NL - 1], P.cinv, P.nc, P.ldc, rr);
  if (!grid_barrier(cnt, gen, nb, P.err)) return false;
  pcg_mark(tm, ph++, P.timing);
  for (int l = NL - 2; l >= 0; --l) {
    const AmgLevelDev& L = P.L[l];
    prolong_from_r<R>(L, P.L[l + 1], rr);
    if (!grid_barrier(cnt, gen, nb, P.err)) return false;
    pcg_mark(tm, ph++, P.timing);
    post_c_r<R>(L, rr);
    if (!grid_barrier(cnt, gen, nb, P.err)) return false;
    pcg_mark(tm, ph++, P.timing);
    double rz = 0.0, wz = 0.0;
    post_d_r<R>(L, rr, P.r, P.diag, rz, wz, l == 0);
    if (l == 0) cta_partial(P.part, slot, rz, wz, 0.0, 0.0, sh);
    if (!grid_barrier(cnt, gen, nb, P.err)) return false;
    pcg_mark(tm, ph++, P.timing);
  }
  return true;
}

// k_pcg_amg on R identical blocks: one CG on the block-diagonal system (the scalars are those of
// the whole system, as for a disjoint union), with the block's matrix and hierarchy stored once.
// Per-row data (rsum, diag, level dinv) are those of block row i (identical blocks); b, x,
// y, bh are indexed in block order (r n + i), the work vectors r, p, q and the level vectors
// interleaved (i R + r).
template <class TV, int R>
__global__ void __launch_bounds__(PCG_BLOCK_R, PCG_CTAS_PER_SM) k_pcg_amg_r(PcgParams<TV> P) {
  unsigned long long tm = 0ull;
  __shared__ double sh[160];
  const unsigned nb = gridDim.x;
  const int lane = threadIdx.x & 31;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (gridDim.x * (int64_t)blockDim.x) >> 5;
  unsigned int* cnt = P.bar;
  unsigned int* gen = P.bar + 1;
  const int64_t n = P.n;
  float* b0 = P.L[0].b;
  float* db0 = P.L[0].db;
  const float* dinv0 = P.L[0].dinv;
  double tot[4];
  double meanb = 0.0;
  if (P.project && !P.bh_given) {
    double part = 0.0;
    PCG_ROWS_BEGIN
#pragma unroll
      for (int r = 0; r < R; ++r) part += static_cast<double>(P.b[r * n + row]);
    PCG_ROWS_END
    cta_partial(P.part, 0, part, 0.0, 0.0, 0.0, sh);
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
    cta_total(P.part, 0, tot, sh);
    meanb = tot[0] / static_cast<double>(R * n);
  }
  {
    double bb = 0.0;
    PCG_ROWS_BEGIN
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int64_t j = r * n + row;
        double bv;
        if (P.bh_given) {
          bv = P.bh[j];
        } else {
          bv = static_cast<double>(P.b[j]) - meanb;
          P.bh[j] = bv;
        }
        if (!P.warm) P.y[j] = 0.0;
        bb += bv * bv;
      }
    PCG_ROWS_END
    cta_partial(P.part, 1, bb, 0.0, 0.0, 0.0, sh);
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
  }
  cta_total(P.part, 1, tot, sh);
  const double bb = tot[0];
  if (P.warm && !(bb > 0.0)) {  // b = 0: the solution is 0
    PCG_ROWS_BEGIN
#pragma unroll
      for (int r = 0; r < R; ++r) P.y[r * n + row] = 0.0;
    PCG_ROWS_END
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
  }
  const double tol2 = fmax(P.rtol * P.rtol * bb, P.atol * P.atol);
  int total = 0, outers = 0;
  double rr = 0.0, rr0 = -1.0;
  for (int outer = 0; outer < P.max_outer; ++outer) {
    ++outers;
    // true residual r = bh - A y (FP64) of every block, its norm, r -> level-0 rhs
    {
      double rh = 0.0;
      const uint64_t pst = l2_policy_stream(), pkeep = l2_policy_keep();
      PCG_SLICES_BEGIN
        double acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = 0.0;
        int k = 0;
        for (; k + 2 <= width; k += 2) {
          const int64_t idx = base + ((int64_t)k << 5) + lane;
          const double v0 = ld_hint(P.a64 + idx, pst), v1 = ld_hint(P.a64 + idx + 32, pst);
          const int32_t c0 = ld_hint(P.col + idx, pkeep), c1 = ld_hint(P.col + idx + 32, pkeep);
#pragma unroll
          for (int r = 0; r < R; ++r) acc[r] += v0 * P.y[r * n + c0] + v1 * P.y[r * n + c1];
        }
        if (k < width) {
          const int64_t idx = base + ((int64_t)k << 5) + lane;
          const double v = ld_hint(P.a64 + idx, pst);
          const int32_t c = ld_hint(P.col + idx, pkeep);
#pragma unroll
          for (int r = 0; r < R; ++r) acc[r] += v * P.y[r * n + c];
        }
        const float di0 = dinv0[row];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const double rv = P.bh[r * n + row] - acc[r];
          const int64_t j = row * R + r;
          P.r[j] = rv;
          const float rf = static_cast<float>(rv);
          b0[j] = rf;
          db0[j] = di0 * rf;
          rh += rv * rv;
        }
      PCG_SLICES_END
      cta_partial(P.part, 0, rh, 0.0, 0.0, 0.0, sh);
      if (!grid_barrier(cnt, gen, nb, P.err)) return;
      pcg_mark(tm, 30, P.timing);
    }
    cta_total(P.part, 0, tot, sh);
    rr = tot[0];
    if (rr0 < 0.0) rr0 = rr;
    if (rr <= tol2 || total >= P.maxit) break;
    const double rr_start = rr;
    double rz_old = 1.0;
    for (int it = 0;; ++it) {
      if (!vcycle_r<TV, R>(P, 2, sh, tm)) return;
      cta_total(P.part, 2, tot, sh);
      const double rz = tot[0];
      const double c = P.project && P.ww > 0.0 ? tot[1] / P.ww : 0.0;
      const double beta = it == 0 ? 0.0 : rz / rz_old;
      const float* u0 = P.L[0].x;  // u of every block (interleaved)
      double pq = 0.0;
      const uint64_t pkeep = l2_policy_keep();
      PCG_SLICES_BEGIN
        float uf[R];
        load_r<R>(u0, row, uf);
        const double rs = P.rsum[row];
        double ui[R], acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          ui[r] = static_cast<double>(uf[r]);
          acc[r] = 0.0;
        }
        for (int k = 0; k < width; k += 4) {  // rounds of four columns, the last predicated
          const int64_t i0 = base + ((int64_t)k << 5) + lane;
          float w[4];
          int32_t cc[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const bool in = k + u < width;
            w[u] = in ? ld_hint(P.a32 + i0 + 32 * u, pkeep) : 0.0f;
            cc[u] = in ? ld_hint(P.col + i0 + 32 * u, pkeep) : 0;
          }
          float g[4][R];
#pragma unroll
          for (int u = 0; u < 4; ++u) load_r<R>(u0, cc[u], g[u]);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (k + u < width) {
#pragma unroll
              for (int r = 0; r < R; ++r)
                acc[r] += static_cast<double>(w[u]) * (static_cast<double>(g[u][r]) - ui[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int64_t j = row * R + r;
          const double av = acc[r] + rs * ui[r];
          const double pv = (ui[r] - c) + (it == 0 ? 0.0 : beta * P.p[j]);
          const double qv = av + (it == 0 ? 0.0 : beta * P.q[j]);
          P.p[j] = pv;
          P.q[j] = qv;
          pq += pv * qv;
        }
      PCG_SLICES_END
      cta_partial(P.part, 3, pq, 0.0, 0.0, 0.0, sh);
      if (!grid_barrier(cnt, gen, nb, P.err)) return;
      pcg_mark(tm, 28, P.timing);
      cta_total(P.part, 3, tot, sh);
      const double pqt = tot[0];
      if (!(pqt > 0.0) || !(rz > 0.0)) break;
      const double alpha = rz / pqt;
      double rh = 0.0;
      PCG_ROWS_BEGIN
        const float di0 = dinv0[row];
        double pv[R], rv[R], qv[R];
        load_r64<R>(P.p, row, pv);
        load_r64<R>(P.r, row, rv);
        load_r64<R>(P.q, row, qv);
        float bf[R], dbf[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          P.y[r * n + row] += alpha * pv[r];
          rv[r] -= alpha * qv[r];
          const float rf = static_cast<float>(rv[r]);
          bf[r] = rf;
          dbf[r] = di0 * rf;
          rh += rv[r] * rv[r];
        }
        store_r64<R>(P.r, row, rv);
        store_r<R>(b0, row, bf);
        store_r<R>(db0, row, dbf);
      PCG_ROWS_END
      cta_partial(P.part, 0, rh, 0.0, 0.0, 0.0, sh);
      if (!grid_barrier(cnt, gen, nb, P.err)) return;
      pcg_mark(tm, 29, P.timing);
      cta_total(P.part, 0, tot, sh);
      rr = tot[0];
      ++total;
      rz_old = rz;
      if (pcg_stop(rr, rr_start, tol2) || total >= P.maxit) break;
    }
  }
  double mx = 0.0;
  if (P.project) {
    double sx = 0.0;
    PCG_ROWS_BEGIN
#pragma unroll
      for (int r = 0; r < R; ++r) sx += P.y[r * n + row];
    PCG_ROWS_END
    cta_partial(P.part, 1, sx, 0.0, 0.0, 0.0, sh);
    if (!grid_barrier(cnt, gen, nb, P.err)) return;
    cta_total(P.part, 1, tot, sh);
    mx = tot[0] / static_cast<double>(R * n);
  }
  PCG_ROWS_BEGIN
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int64_t j = r * n + row;
      const double xv = P.y[j] - mx;
      P.x[j] = static_cast<TV>(xv);
      P.y[j] = xv;
    }
  PCG_ROWS_END
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *P.iters = total;
    *P.resid = bb > 0.0 ? sqrt(rr / bb) : 0.0;
    atomicAdd(P.iters_acc, (unsigned long long)total);
    atomicAdd(P.iters_acc + 1, (unsigned long long)outers);
    atomicAdd(P.iters_acc + 2, 1ull);
    if (bb > 0.0) {
      atomicAdd(P.res_acc, sqrt(fmax(rr0, 0.0) / bb));
      atomicAdd(P.res_acc + 1, sqrt(rr / bb));
    }
  }
}

}  // namespace

// ------------------------------------------------------------------ host entry
template <class TM>
void CgSystem<TM>::enable_amg(const HostSell& hs, const std::vector<int64_t>& rowptr, const std::vector<int32_t>& col,
                              const std::vector<double>& a, const std::vector<double>& d, bool singular,
                              cudaStream_t s) {
  const int64_t n = n1;  // the stored block (reps copies of it form the system)
  CsrHost Ah;
  Ah.n = n;
  Ah.ncols = n;
  Ah.rp = rowptr;
  Ah.ci = col;
  Ah.v.resize(a.size());
  for (int64_t i = 0; i < n; ++i)
    for (int64_t k = rowptr[i]; k < rowptr[i + 1]; ++k) Ah.v[k] = a[k] / std::sqrt(d[i] * d[col[k]]);
  std::vector<double> w(n);
  double ww = 0.0;
  for (int64_t i = 0; i < n; ++i) {
    w[i] = std::sqrt(d[i]);
    ww += d[i];
  }
  ww *= reps;  // the null vector of the whole system repeats w in every block
  AmgHost h;
  amg_build(Ah, w, singular, AmgOptions{}, h);
  if (h.lv.size() < 2) {  // no coarsening possible: keep the Jacobi solver
    amg.reset();
    return;
  }
  // unscaled FP32 values on the SELL pattern and FP64 row sums (difference-form SpMV); the
  // finest level of the cycle uses the same values
  {
    std::vector<float> v(P.len, 0.0f);
    std::vector<double> rs(n, 0.0);
    for (int64_t i = 0; i < n; ++i)
      for (int64_t k = rowptr[i]; k < rowptr[i + 1]; ++k) {
        rs[i] += a[k];
        if (hs.map[k] >= 0) v[hs.map[k]] = static_cast<float>(a[k]);
      }
    amg_a32.upload(v, s);
    amg_rsum.upload(rs, s);
  }
  // level 0 in the unscaled space: D^-1 of A, P_0 = D^-1/2 P^_0, R_0 = P^_0^T D^-1/2
  {
    AmgHostLevel& L0 = h.lv[0];
    for (int64_t i = 0; i < n; ++i) L0.dinv[i] = 1.0 / d[i];
    for (int64_t i = 0; i < n; ++i)
      for (int64_t k = L0.P.rp[i]; k < L0.P.rp[i + 1]; ++k) L0.P.v[k] /= std::sqrt(d[i]);
    for (int64_t k = 0; k < static_cast<int64_t>(L0.R.v.size()); ++k) L0.R.v[k] /= std::sqrt(d[L0.R.ci[k]]);
  }
  int dev;
  SPX_CUDA(cudaGetDevice(&dev));
  amg_grid = num_sms(dev) * PCG_CTAS_PER_SM;
  amg = std::make_unique<AmgDevice>();
  amg->upload(h, s, P.slice_ptr.p, P.col.p, amg_a32.p, P.nslices, reps, amg_grid);
  amg_ww = ww;
  amg_singular = singular;
  if (!y64.n) {
    y64.alloc(this->n);
    y64.zero(s);
  }
  if (!bh64.n) bh64.alloc(this->n);
  amg_work.alloc(3 * static_cast<size_t>(this->n));
  amg_work.zero(s);
  {  // unscaled FP64 values (true residual)
    std::vector<double> v(P.len, 0.0);
    for (int64_t k = 0; k < static_cast<int64_t>(a.size()); ++k)
      if (hs.map[k] >= 0) v[hs.map[k]] = a[k];
    vals64.upload(v, s);
    vals.release();  // the scaled values and vectors belong to the Jacobi solvers
    work.release();
  }
  SPX_CHECK(reps == 1 || reps == 2 || reps == 4 || reps == 8, "repeated blocks: 1, 2, 4 or 8");
  int per_sm = 0;
  if (reps == 1) {
    plan_resident();
    for (const void* kk : {reinterpret_cast<const void*>(k_pcg_amg<double>), reinterpret_cast<const void*>(k_pcg_amg<float>)})
      SPX_CUDA(cudaFuncSetAttribute(kk, cudaFuncAttributeMaxDynamicSharedMemorySize, PCG_DYN_MAX));
    SPX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pcg_amg<double>, PCG_BLOCK, amg->smem_bytes));
    SPX_CHECK(per_sm >= PCG_CTAS_PER_SM, "AMG PCG kernel cannot be resident");
  }
  if (reps > 1) {
    const void* kr = reps == 2 ? reinterpret_cast<const void*>(k_pcg_amg_r<double, 2>)
                     : reps == 4 ? reinterpret_cast<const void*>(k_pcg_amg_r<double, 4>)
                                 : reinterpret_cast<const void*>(k_pcg_amg_r<double, 8>);
    // the coarse phase stages the R right-hand sides in dynamic shared memory
    const size_t dyn = static_cast<size_t>(amg->nc) * reps * sizeof(float);
    SPX_CHECK(dyn <= 200 * 1024, "AMG coarsest level too large for the repeated-block kernel");
    const void* kall[] = {reinterpret_cast<const void*>(k_pcg_amg_r<double, 2>),
                          reinterpret_cast<const void*>(k_pcg_amg_r<double, 4>),
                          reinterpret_cast<const void*>(k_pcg_amg_r<double, 8>),
                          reinterpret_cast<const void*>(k_pcg_amg_r<float, 2>),
                          reinterpret_cast<const void*>(k_pcg_amg_r<float, 4>),
                          reinterpret_cast<const void*>(k_pcg_amg_r<float, 8>)};
    for (const void* kk : kall)
      SPX_CUDA(cudaFuncSetAttribute(kk, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(dyn)));
    SPX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kr, PCG_BLOCK_R, dyn));
    SPX_CHECK(per_sm >= PCG_CTAS_PER_SM, "AMG PCG kernel (repeated blocks) cannot be resident");
  }
  {
    int64_t keep = P.len * static_cast<int64_t>(sizeof(float) + sizeof(int32_t));  // level 0 (shared pattern)
    for (int l = 1; l + 1 < amg->nlev; ++l) keep += amg->A[l].len * static_cast<int64_t>(sizeof(float) + sizeof(int32_t));
    keep += amg->cinv.bytes();  // the dense coarsest inverse
    reserve_persisting_l2(keep + keep / 8, dev);
  }
  if (part.n < 4 * 4 * static_cast<size_t>(amg_grid)) part.alloc(4 * 4 * static_cast<size_t>(amg_grid));
  SPX_CUDA(cudaStreamSynchronize(s));
}

// Shared memory of k_pcg_amg, finest level first: the slice bounds of a level (4 bytes a slice),
// then as many of its entries (FP32 value and column) as still fit.  400x400x2 film: all of
// level 0 (165 KB a CTA) and part of level 1.
template <class TM>
void CgSystem<TM>::plan_resident() {
  AmgDevice& A = *amg;
  A.res.assign(A.nlev, AmgResident{-1, 0, 0, 0, 0, 0});
  int64_t pos = 0;  // words
  const int64_t lim = PCG_DYN_MAX / 4;
  for (int l = 0; l + 1 < A.nlev; ++l) {
    const int64_t words = (A.cnt[l] + 1 + 3) / 4 * 4;
    const int64_t rwords = ((A.sizes[l + 1] + amg_grid - 1) / amg_grid + 1 + 3) / 4 * 4;
    if (pos + 2 * words + rwords > lim / 4) break;  // a level of thousands of slices a CTA streams
    A.res[l].off = static_cast<int32_t>(pos);
    A.res[l].poff = static_cast<int32_t>(pos + words);
    A.res[l].roff = static_cast<int32_t>(pos + 2 * words);
    pos += 2 * words + rwords;
  }
  for (int l = 0; l + 1 < A.nlev && A.res[l].off >= 0; ++l) {
    const int64_t cap = std::min<int64_t>(A.need[l], (lim - pos) / 2 / 32 * 32);
    A.res[l].val = static_cast<int32_t>(pos);
    A.res[l].col = static_cast<int32_t>(pos + cap);
    A.res[l].cap = static_cast<int32_t>(cap);
    pos += 2 * cap;
  }
  A.smem_bytes = static_cast<size_t>(pos) * 4;
}

template <class TM>
template <class TV>
void CgSystem<TM>::launch_amg(const TV* b, TV* x, double rtol, double atol, int maxit, bool warm, bool project,
                              cudaStream_t st, bool bh_given) {
  PcgParams<TV> q;
  q.n = n1; q.nslices = P.nslices; q.sp = P.slice_ptr.p; q.col = P.col.p; q.reps = reps;
  q.a64 = vals64.p; q.a32 = amg_a32.p; q.rsum = amg_rsum.p; q.diag = diag64.p;
  q.b = b; q.x = x;
  q.bh = bh64.p; q.y = y64.p;
  q.r = amg_work.p; q.p = amg_work.p + n; q.q = amg_work.p + 2 * n;
  q.part = part.p; q.bar = bar.p; q.err = err.p; q.iters = iters.p; q.resid = resid.p;
  q.iters_acc = iters_acc.p; q.res_acc = res_acc.p;
  q.rtol = rtol; q.atol = atol; q.ww = amg_singular ? amg_ww : 0.0;
  q.maxit = maxit; q.max_outer = max_outer; q.warm = warm ? 1 : 0; q.project = project ? 1 : 0;
  q.bh_given = bh_given ? 1 : 0;
  q.nlev = amg->nlev;
  for (int l = 0; l < amg->nlev; ++l) {
    q.L[l] = amg->lv[l];
    q.R[l] = amg->res[l];
  }
  q.cinv = amg->cinv.p; q.nc = amg->nc; q.ldc = amg->ldc;
  q.timing = g_pcg_timing.load(std::memory_order_relaxed);
  void* args[] = {&q};
  void* k = reinterpret_cast<void*>(k_pcg_amg<TV>);
  if (reps == 2) k = reinterpret_cast<void*>(k_pcg_amg_r<TV, 2>);
  if (reps == 4) k = reinterpret_cast<void*>(k_pcg_amg_r<TV, 4>);
  if (reps == 8) k = reinterpret_cast<void*>(k_pcg_amg_r<TV, 8>);
  const size_t dyn = reps > 1 ? static_cast<size_t>(amg->nc) * reps * sizeof(float) : amg->smem_bytes;
  SPX_CUDA(cudaLaunchCooperativeKernel(k, dim3(amg_grid), dim3(reps > 1 ? PCG_BLOCK_R : PCG_BLOCK), args, dyn, st));
}

// per-slot sums (ns) and counts of the phase timing marks since the last call
void pcg_phase_times(double* ns32, int64_t* n32) {
  unsigned long long a[32], b[32], z[32] = {};
  SPX_CUDA(cudaDeviceSynchronize());
  SPX_CUDA(cudaMemcpyFromSymbol(a, g_pcg_phase_ns, sizeof(a)));
  SPX_CUDA(cudaMemcpyFromSymbol(b, g_pcg_phase_n, sizeof(b)));
  SPX_CUDA(cudaMemcpyToSymbol(g_pcg_phase_ns, z, sizeof(z)));
  SPX_CUDA(cudaMemcpyToSymbol(g_pcg_phase_n, z, sizeof(z)));
  for (int i = 0; i < 32; ++i) {
    ns32[i] = static_cast<double>(a[i]);
    n32[i] = static_cast<int64_t>(b[i]);
  }
}

template void CgSystem<double>::enable_amg(const HostSell&, const std::vector<int64_t>&, const std::vector<int32_t>&,
                                           const std::vector<double>&, const std::vector<double>&, bool,
                                           cudaStream_t);
template void CgSystem<float>::enable_amg(const HostSell&, const std::vector<int64_t>&, const std::vector<int32_t>&,
                                          const std::vector<double>&, const std::vector<double>&, bool,
                                          cudaStream_t);
template void CgSystem<double>::launch_amg<double>(const double*, double*, double, double, int, bool, bool,
                                                   cudaStream_t, bool);
template void CgSystem<float>::launch_amg<double>(const double*, double*, double, double, int, bool, bool,
                                                  cudaStream_t, bool);
template void CgSystem<float>::launch_amg<float>(const float*, float*, double, double, int, bool, bool,
                                                 cudaStream_t, bool);

}  // namespace spx
