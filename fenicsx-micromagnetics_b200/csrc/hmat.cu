// H-matrix apply: y = P^-1 [diag o x~ + Near x~ + sum_b U_b (V_b x~_{J_b})],  x~ = x[perm]
// (HMatrixGPUPackedFused.matvec, lindholm_hmatrix_gpu/backend_fused.py:496-512).
//
// B200 layout (built by pack() from the FP64 pools of the builder, in the storage type TF of
// the far factors -- FP64, FP32 or BF16 -- and TN of the near tiles -- FP64 or FP32):
//   * row segments: the leaf clusters in permutation order, split into pieces of at most
//     64 rows; every output row belongs to exactly one segment.
//   * V_b^T of each far block: n rows of ldk = k rounded up to 16 bytes (row c holds
//     V_b[0..k-1, c]), cut into units of at most ~16 KB of rows.
//   * U_b of each far block, cut at the segments it covers: per segment a tile of k rows of
//     ld = rows rounded up to a 16-byte multiple (row q holds U[rows, q]).
//   * near blocks, cut the same way: per segment a tile of n columns of ld entries.
// Every tile and row starts 16-byte aligned and is zero padded, so all factor traffic is
// 16-byte vector loads of contiguous memory.
//
// Kernels (no atomics on data, every output written by exactly one warp or CTA):
//   k_hgather : x~[i] = src[g(perm[i])]             (fused boundary gather + perm)
//   k_far_z   : z_b = V_b x~_{J_b} = sum_c x~_c V_b^T[c, :].  Warps over contiguous, byte-balanced
//               ranges of tiles; lanes = (16-byte vector of outputs q, phase over rows c),
//               accumulating in registers across the tiles of a block; at the block's last tile
//               in the warp a shuffle sum over the phases writes z_b.  A block shared by several
//               warps (only at range ends) adds the warps' partials through an arrival counter:
//               the last arriving warp sums them in contributor order and resets the counter,
//               so z does not depend on scheduling.
//   k_rows    : CTAs over contiguous, byte-balanced ranges of the row segments' tiles (U tiles
//               with z_b, near tiles with x~), lanes over 16-byte row vectors x phases over the
//               tile rows, then a fixed-order sum over warps, + diag o x~, scattered to
//               dst[g(perm[i])]; segments cut by a range end are joined like the blocks.
// Each warp keeps its next tile moving into L2 with cp.async.bulk.prefetch.L2, and each kernel
// starts that while the one before it finishes (programmatic dependent launch).
// Near tiles use compensated (Kahan) accumulation when FP32 accumulates BF16/FP32 data in
// the mixed-precision form.
#include <algorithm>
#include <mutex>
#include <string>

#include <cuda_fp16.h>

#include "bulk.cuh"
#include "hmat.cuh"

namespace spx {

template <class T> __device__ __forceinline__ T from_d(double v) { return static_cast<T>(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_d<__nv_bfloat16>(double v) {
  return __float2bfloat16_rn(static_cast<float>(v));
}
template <class T> __device__ __forceinline__ double to_d(T v) { return static_cast<double>(v); }
template <> __device__ __forceinline__ double to_d<__nv_bfloat16>(__nv_bfloat16 v) {
  return static_cast<double>(__bfloat162float(v));
}
template <class A, class T> __device__ __forceinline__ A cvt(T v) { return static_cast<A>(v); }
template <> __device__ __forceinline__ float cvt<float, __nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ double cvt<double, __nv_bfloat16>(__nv_bfloat16 v) {
  return static_cast<double>(__bfloat162float(v));
}


// ------------------------------------------------------------------ packing
namespace {
constexpr int Z_WARPS = 8;      // warps per CTA and CTAs per SM of the multi-state far_z
constexpr int Z_CTAS_PER_SM = 4;
constexpr int SEG_MAX = 64;     // rows per segment
inline int64_t round_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }
}  // namespace

// dst[q * ld + r] = pool[src + q * sq + r * sr] * (scaled by qscale[qs + q] when qs >= 0, or
// by rscale[qs + r] when rs != 0) for r < nr, 0 for nr <= r < ld, q < nq
struct PackJob {
  int64_t src, dst;
  int32_t nq, nr, ld, sq, sr;
  int64_t qs = -1;  // first scale factor of this job (-1: none)
  int32_t rs = 0;   // 1: the scale runs along r instead of q
};
template <class T> __device__ __forceinline__ T from_d_s(double v) { return from_d<T>(v); }
template <> __device__ __forceinline__ __half from_d_s<__half>(double v) { return __double2half(v); }
template <class T>
__global__ void k_pack(const PackJob* __restrict__ jobs, int64_t njobs, const double* __restrict__ pool,
                       const double* __restrict__ scale, T* __restrict__ out) {
  for (int64_t jb = blockIdx.x; jb < njobs; jb += gridDim.x) {
    const PackJob j = jobs[jb];
    const int64_t L = static_cast<int64_t>(j.nq) * j.ld;
    for (int64_t e = threadIdx.x; e < L; e += blockDim.x) {
      const int64_t q = e / j.ld, r = e - q * j.ld;
      double v = r < j.nr ? pool[j.src + q * j.sq + r * j.sr] : 0.0;
      if (j.qs >= 0 && r < j.nr) v *= scale[j.qs + (j.rs ? r : q)];
      out[j.dst + e] = from_d_s<T>(v);
    }
  }
}

// ------------------------------------------------------------------ apply kernels
template <class TS, class TX>
__global__ void k_hgather(int64_t Nb, const TS* __restrict__ src, const int32_t* __restrict__ gidx,
                          const int32_t* __restrict__ perm, TX* __restrict__ xp) {
  pdl_trigger();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= Nb) return;
  const int32_t b = perm[i];
  const int64_t o = gidx ? gidx[b] : b;
  xp[i] = static_cast<TX>(src[o]);
}

// 16-byte vector loads of far factors
template <class TF> struct V16;
template <> struct V16<double> { using T = double2; static constexpr int E = 2; };
template <> struct V16<float> { using T = float4; static constexpr int E = 4; };
template <> struct V16<__nv_bfloat16> { using T = uint4; static constexpr int E = 8; };
template <> struct V16<__half> { using T = uint4; static constexpr int E = 8; };

template <class TA, class TF>
__device__ __forceinline__ void v16_elems(const typename V16<TF>::T& v, TA out[V16<TF>::E]);
template <>
__device__ __forceinline__ void v16_elems<double, double>(const double2& v, double out[2]) { out[0] = v.x; out[1] = v.y; }
template <>
__device__ __forceinline__ void v16_elems<float, double>(const double2& v, float out[2]) {
  out[0] = static_cast<float>(v.x); out[1] = static_cast<float>(v.y);
}
template <>
__device__ __forceinline__ void v16_elems<double, float>(const float4& v, double out[4]) {
  out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
}
template <>
__device__ __forceinline__ void v16_elems<float, float>(const float4& v, float out[4]) {
  out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
}
template <class TA>
__device__ __forceinline__ void bf16x8(const uint4& v, TA out[8]) {
  const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    out[2 * q] = static_cast<TA>(__uint_as_float(w[q] << 16));
    out[2 * q + 1] = static_cast<TA>(__uint_as_float(w[q] & 0xffff0000u));
  }
}
template <class TA>
__device__ __forceinline__ void h16x8(const uint4& v, TA out[8]) {
  const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[q]));
    out[2 * q] = static_cast<TA>(f.x);
    out[2 * q + 1] = static_cast<TA>(f.y);
  }
}
template <>
__device__ __forceinline__ void v16_elems<double, __half>(const uint4& v, double out[8]) { h16x8<double>(v, out); }
template <>
__device__ __forceinline__ void v16_elems<float, __half>(const uint4& v, float out[8]) { h16x8<float>(v, out); }
template <>
__device__ __forceinline__ void v16_elems<double, __nv_bfloat16>(const uint4& v, double out[8]) { bf16x8<double>(v, out); }
template <>
__device__ __forceinline__ void v16_elems<float, __nv_bfloat16>(const uint4& v, float out[8]) { bf16x8<float>(v, out); }



// asynchronous prefetch of a contiguous range into L2 (cp.async.bulk.prefetch.L2; 16-byte
// aligned address, size a multiple of 16)
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// What bounds the apply: with FP64 factors HBM (film of 400 cubes a side, 13.8 GB: 6.2 TB/s, 0.94 of
// the copy rate).  FP32 (6.9 GB, 4.8 TB/s) and BF16 factors (about 3.9 GB, 2.8 TB/s) take nearly the
// same time as each other at that size, so there it goes with the entries, not with the bytes (which
// part of an entry's chain of loads, conversion and sum is not settled: one XOR in place of the FMAs
// changes neither kernel's time).  32 warps per SM with four 16-byte loads of a lane in flight and the
// next tile of each warp on its way into L2.  Tiles of 16 KB cost FP64 factors 18 % and FP32 ones
// 1-13 %, 2 KB tiles 6-17 %; three CTAs with six loads a lane FP32 8 %.
// us per product (CTA per row segment, power-of-two lane split, 16 KB units -> this), films of 24,
// 48, 100, 150, 200, 400 cubes a side: FP32 31.8 -> 24.2, 42.4 -> 29.1, 95 -> 67.6, 167 -> 152,
// 296 -> 270, 1436 -> 1443 (no gain there); FP64 29.6 -> 23.5, 43.2 -> 29.4, 126 -> 102, 260 -> 228,
// 465 -> 423, 2359 -> 2243; BF16 28.7 -> 29.6, 44.0 -> 33.5, 86 -> 69, 157 -> 138, 280 -> 249, 1417 -> 1384.
constexpr int ST_WARPS = 8;          // warps per CTA
constexpr int ST_CTAS_PER_SM = 4;
constexpr int ST_TILE = 4096;        // bytes of a tile
constexpr int ST_THREADS = ST_WARPS * 32;
constexpr int ST_U = 4;              // 16-byte loads of a lane in flight

// acc[t] += sum over rows q < len of tile[q][vl E + t] v[q].  Lanes: the nv 16-byte vectors of a row
// times P = 32 / nv phases over the rows (lane = ph nv + vl; lanes past P nv idle), ST_U rows of a
// phase in flight.  A split into powers of two (nv rounded up) would leave a quarter of the lanes
// idle at rank 24, three eighths at 40 rows.
template <class T, class TA, class TV, int E, bool KAHAN>
__device__ __forceinline__ void tile_dot(const T* tile_t, const TV* v, int len, int nv, int P, int vl, int ph,
                                         TA (&acc)[E], TA (&cmp)[E]) {
  using VT = typename V16<T>::T;
  const VT* tile = reinterpret_cast<const VT*>(tile_t) + ph * nv + vl;
  const int st = P * nv;
  v += ph;
  auto add = [&](const VT& w, TA a) {
    TA e[E];
    v16_elems<TA, T>(w, e);
#pragma unroll
    for (int t = 0; t < E; ++t) {
      if (KAHAN) {
        const TA y = e[t] * a - cmp[t];
        const TA s = acc[t] + y;
        cmp[t] = (s - acc[t]) - y;
        acc[t] = s;
      } else {
        acc[t] += e[t] * a;
      }
    }
  };
  int q = ph;
  for (; q + (ST_U - 1) * P < len; q += ST_U * P) {
    VT w[ST_U];
    TA a[ST_U];
#pragma unroll
    for (int u = 0; u < ST_U; ++u) {
      w[u] = tile[u * st];
      a[u] = static_cast<TA>(v[u * P]);
    }
#pragma unroll
    for (int u = 0; u < ST_U; ++u) add(w[u], a[u]);
    tile += ST_U * st;
    v += ST_U * P;
  }
  for (; q < len; q += P) {
    add(*tile, static_cast<TA>(*v));
    tile += st;
    v += P;
  }
}
// the sum over the phases, in lanes of phase 0: one after the other for a few phases, else a tree
// (halves of the next power of two first)
template <class TA>
__device__ __forceinline__ TA phase_sum(TA a, int nv, int P, int ph) {
  const int lane = threadIdx.x & 31;
  TA y = a;
  if (P <= 6) {  // uniform
    for (int p = 1; p < P; ++p) y += __shfl_sync(0xffffffffu, a, lane + p * nv);
    return y;
  }
  for (int s = 16; s > 0; s >>= 1)
    if (s < P) {
      const TA t = __shfl_sync(0xffffffffu, y, lane + s * nv);
      if (ph < s && ph + s < P) y += t;
    }
  return y;
}

// z_b = V_b x~: tiles of a block's V^T dealt to warps in contiguous ranges of about equal bytes.
template <class TF, class TA>
__global__ void __launch_bounds__(ST_THREADS, ST_CTAS_PER_SM)
    k_far_z(const StUnit* __restrict__ units, const int32_t* __restrict__ warp_first, int nwarps,
            const TF* __restrict__ F, const TA* __restrict__ xp, TA* __restrict__ z, TA* __restrict__ zpart,
            const FarGroup* __restrict__ groups, unsigned int* __restrict__ gcnt, const double* __restrict__ zscale) {
  constexpr int E = V16<TF>::E;
  pdl_trigger();
  const int lane = threadIdx.x & 31, wg = blockIdx.x * ST_WARPS + (threadIdx.x >> 5);
  if (wg >= nwarps) return;
  int u = warp_first[wg];
  const int u1 = warp_first[wg + 1];
  StUnit nxt;
  if (u < u1) {  // the factors do not depend on the kernel before; x~ does
    nxt = units[u];
    if (lane == 0) prefetch_l2(F + nxt.voff, static_cast<uint32_t>(nxt.nc) * nxt.ldk * sizeof(TF));
  }
  pdl_wait();
  TA acc[E], cmp[E];
#pragma unroll
  for (int t = 0; t < E; ++t) acc[t] = TA(0);
  for (; u < u1; ++u) {
    const StUnit U = nxt;
    if (u + 1 < u1) nxt = units[u + 1];  // descriptor of the next tile in flight
    const int nvq = U.ldk / E, P = U.phases;  // nvq <= 32
    const int ph = (lane * U.magic) >> 16, vl = lane - ph * nvq;  // lane / nvq
    if (ph < P) tile_dot<TF, TA, TA, E, false>(F + U.voff, xp + U.xc, U.nc, nvq, P, vl, ph, acc, cmp);
    if (lane == 0 && u + 1 < u1)  // the next tile into L2
      prefetch_l2(F + nxt.voff, static_cast<uint32_t>(nxt.nc) * nxt.ldk * sizeof(TF));
    const int fl = U.flags;
    if (fl == 0) continue;
    // the block ends in this warp: sum over the phases, write its k rows
#pragma unroll
    for (int t = 0; t < E; ++t) acc[t] = phase_sum(acc[t], nvq, P, ph);
    TA* out = fl == 1 ? z : zpart;
    if (ph == 0) {
#pragma unroll
      for (int t = 0; t < E; ++t) {
        const int q = vl * E + t;
        if (q < U.k) {
          TA v = acc[t];
          if (zscale && fl == 1) v *= static_cast<TA>(zscale[U.zout + q]);
          out[U.zout + q] = v;
        }
      }
    }
#pragma unroll
    for (int t = 0; t < E; ++t) acc[t] = TA(0);
    if (fl == 2) {  // block shared between warps: the last contributor sums the partials in order
      __threadfence();
      __syncwarp();
      const FarGroup Gp = groups[U.grp];
      unsigned last = 0;
      if (lane == 0) last = atomicAdd(gcnt + U.grp, 1u) == static_cast<unsigned>(Gp.ncontrib) - 1u ? 1u : 0u;
      last = __shfl_sync(0xffffffffu, last, 0);
      if (last) {
        __threadfence();
        for (int q = lane; q < Gp.k; q += 32) {
          TA sum = TA(0);
          for (int cc = 0; cc < Gp.ncontrib; ++cc) sum += __ldcg(zpart + Gp.pbase + cc * U.ldk + q);
          if (zscale) sum *= static_cast<TA>(zscale[Gp.zdst + q]);
          z[Gp.zdst + q] = sum;
        }
        if (lane == 0) atomicExch(gcnt + U.grp, 0u);
      }
    }
  }
}

// sum over the phases into the warp's rows of the portion (set: first drain of the portion), and
// clear the accumulators
template <class TA, int E>
__device__ __forceinline__ void tile_drain(TA (&acc)[E], TA (&cmp)[E], int nr, int nv, int P, int vl, int ph, TA* part,
                                           bool set) {
#pragma unroll
  for (int t = 0; t < E; ++t) {
    const TA y = phase_sum(acc[t] - cmp[t], nv, P, ph);
    if (ph == 0 && vl * E + t < nr) {
      TA* p = part + vl * E + t;
      *p = set ? y : *p + y;
    }
    acc[t] = cmp[t] = TA(0);
  }
  __syncwarp();
}

// the chunks c, c + ST_WARPS, ... < end of one type: tile rows times v, into acc
template <class T, class TA, int E, bool KAHAN>
__device__ __forceinline__ void chunks_dot(const StChunk* __restrict__ chunks, int& c, int end, StChunk& nxt, int last,
                                           const T* __restrict__ base, const TA* __restrict__ v, int type, int nv, int P,
                                           int vl, int ph, int lane, TA (&acc)[E], TA (&cmp)[E]) {
  for (; c < end && nxt.type == type; c += ST_WARPS) {
    const StChunk C = nxt;
    if (c + ST_WARPS < last) nxt = chunks[c + ST_WARPS];
    if (lane == 0 && c + ST_WARPS < last && nxt.type == type)  // the next tile into L2
      prefetch_l2(base + nxt.off, static_cast<uint32_t>(nxt.len) * nxt.ld * sizeof(T));
    if (ph < P) tile_dot<T, TA, TA, E, KAHAN>(base + C.off, v + C.src, C.len, nv, P, vl, ph, acc, cmp);
  }
}

// y = diag x~ + U z + Near x~.  Every CTA takes a contiguous range of chunks (tiles, in segment
// order), balanced by bytes over the CTAs whatever the segments' sizes; its warps take the
// range's chunks round-robin.  A portion is the part of a segment inside the range: at its end
// each warp leaves its sums in shared memory, and after a CTA barrier one warp (they take turns)
// adds them in warp order and writes the rows, or, for a segment shared by several CTAs, leaves a
// partial that the last of them adds up in portion order, while the others go on with the next
// portion in the other buffer.  Mbarriers that let a warp run two portions ahead: FP64 2-4 % slower,
// FP32 the same, BF16 1-2 % faster (200 and 400 cubes a side), and a wait that can give up.
template <class TF, class TN, class TA, class TD>
__global__ void __launch_bounds__(ST_THREADS, ST_CTAS_PER_SM) k_rows(
    const StPortion* __restrict__ portions, const int32_t* __restrict__ cta_first, const StChunk* __restrict__ chunks,
    const TF* __restrict__ F, const TN* __restrict__ Nt, const __half* __restrict__ Fh, const TA* __restrict__ z,
    const TA* __restrict__ xp, const double* __restrict__ diag, const int32_t* __restrict__ perm,
    const int32_t* __restrict__ gidx, TD* __restrict__ dst, const TD* __restrict__ add, TD* __restrict__ yb,
    const int2* __restrict__ groups, unsigned int* __restrict__ gcnt, TA* __restrict__ ypart) {
  constexpr int EF = V16<TF>::E, EN = V16<TN>::E, EH = V16<__half>::E;
  constexpr bool KAHAN = sizeof(TA) == sizeof(float) && sizeof(TF) < sizeof(double);
  __shared__ TA part[2][ST_WARPS][SEG_MAX];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p0 = cta_first[blockIdx.x], p1 = cta_first[blockIdx.x + 1];
  if (p0 >= p1) return;  // uniform per CTA
  const int c1 = portions[p1 - 1].c1;
  int c = portions[p0].c0 + warp;
  StChunk nxt;
  if (c < c1) {
    nxt = chunks[c];
    if (lane == 0) {
      const uint32_t n = static_cast<uint32_t>(nxt.len) * nxt.ld;
      if (nxt.type == 0) prefetch_l2(F + nxt.off, n * static_cast<uint32_t>(sizeof(TF)));
      else if (nxt.type == 2) prefetch_l2(Nt + nxt.off, n * static_cast<uint32_t>(sizeof(TN)));
    }
  }
  pdl_wait();  // z and x~ are complete
  for (int p = p0; p < p1; ++p) {
    const StPortion Q = portions[p];
    const int nr = Q.nr;
    const int k = p - p0, b = k & 1;
    TA* mine = part[b][warp];
    bool set = true;
    auto turn = [&](auto typ, auto kah, int type, const auto* base, const TA* v) {
      using T = decltype(typ);
      constexpr int E = V16<T>::E;
      const int nv = (nr + E - 1) / E, P = 32 / nv, ph = lane / nv, vl = lane - ph * nv;
      TA acc[E], cmp[E];
#pragma unroll
      for (int t = 0; t < E; ++t) acc[t] = cmp[t] = TA(0);
      chunks_dot<T, TA, E, decltype(kah)::value>(chunks, c, Q.c1, nxt, c1, base, v, type, nv, P, vl, ph, lane, acc, cmp);
      tile_drain<TA, E>(acc, cmp, nr, nv, P, vl, ph, mine, set);
      set = false;
    };
    turn(TF{}, std::false_type{}, 0, F, z);
    if (Fh && c < Q.c1 && nxt.type == 1) turn(__half{}, std::false_type{}, 1, Fh, z);
    if (c < Q.c1 && nxt.type == 2) turn(TN{}, std::integral_constant<bool, KAHAN>{}, 2, Nt, xp);
    // buffer b is complete; the warp that read it two portions ago has passed the barrier after that
    __syncthreads();
    if (k % ST_WARPS != warp) continue;
    TA y[2] = {TA(0), TA(0)};  // rows lane, lane + 32
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (lane + 32 * h < nr)
        for (int w = 0; w < ST_WARPS; ++w) y[h] += part[b][w][lane + 32 * h];
    if (Q.grp >= 0) {  // segment shared with other CTAs: the last portion adds the partials up
      const int2 G = groups[Q.grp];  // first partial, number of them
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (lane + 32 * h < nr) ypart[static_cast<int64_t>(Q.slot) * SEG_MAX + lane + 32 * h] = y[h];
      __threadfence();
      __syncwarp();
      int last = 0;
      if (lane == 0) last = atomicAdd(gcnt + Q.grp, 1u) == static_cast<unsigned>(G.y) - 1u ? 1 : 0;
      if (!__shfl_sync(0xffffffffu, last, 0)) continue;
      __threadfence();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        y[h] = TA(0);
        if (lane + 32 * h < nr)
          for (int g = 0; g < G.y; ++g) y[h] += __ldcg(ypart + static_cast<int64_t>(G.x + g) * SEG_MAX + lane + 32 * h);
      }
      if (lane == 0) atomicExch(gcnt + Q.grp, 0u);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lane + 32 * h;
      if (r >= nr) continue;
      const int64_t i = Q.r0 + r;
      const int32_t bi = perm[i];
      const int64_t o = gidx ? gidx[bi] : bi;
      const TD yv = static_cast<TD>(y[h] + static_cast<TA>(diag[i]) * xp[i]);
      dst[o] = add ? static_cast<TD>(add[o] + yv) : yv;
      if (yb) yb[bi] = yv;
    }
  }
}

// ------------------------------------------------------------------ host side
namespace {

template <class T>
void run_pack_jobs(const std::vector<PackJob>& jobs, const double* pool, const double* scale, char* out,
                   cudaStream_t s) {
  if (jobs.empty()) return;
  constexpr size_t CH = size_t(1) << 20;
  for (size_t k0 = 0; k0 < jobs.size(); k0 += CH) {
    const size_t c = std::min(CH, jobs.size() - k0);
    DevBuf<PackJob> d;
    d.upload(jobs.data() + k0, c, s);
    const unsigned grid = static_cast<unsigned>(std::min<size_t>(c, 65535));
    k_pack<T><<<grid, 128, 0, s>>>(d.p, static_cast<int64_t>(c), pool, scale, reinterpret_cast<T*>(out));
    SPX_LAUNCH_CHECK();
    SPX_CUDA(cudaStreamSynchronize(s));
  }
}

// far_z units dealt to warps in contiguous ranges of about equal cost; the last unit of a
// block in each warp writes the block (flags 1), or contributes partials to a group (flags 2)
// whose slots start at *ppos.  Every unit of a block with more vectors per row than a warp has
// lanes is a contribution of its own (k_far_z_multi goes over its rows in strips of 32 vectors).
// Returns the warp ranges.
std::vector<int32_t> plan_units(std::vector<FarUnit>& units, size_t elem_bytes, int nsm, int64_t& nw_out,
                                std::vector<FarGroup>& groups, int64_t& ppos) {
  const int64_t nw = std::max<int64_t>(1, std::min<int64_t>(static_cast<int64_t>(nsm) * Z_CTAS_PER_SM * Z_WARPS,
                                                            static_cast<int64_t>(units.size())));
  std::vector<double> cost(units.size() + 1, 0.0);
  for (size_t u = 0; u < units.size(); ++u) {
    const FarUnit& U = units[u];
    cost[u + 1] = cost[u] + static_cast<double>(U.nc) * U.ldk * elem_bytes + 8.0 * U.nc + 512.0;
  }
  std::vector<int32_t> wf(nw + 1, 0);
  {
    size_t u = 0;
    for (int64_t w = 0; w <= nw; ++w) {
      const double target = cost.back() * static_cast<double>(w) / static_cast<double>(nw);
      while (u < units.size() && cost[u] < target) ++u;
      wf[w] = static_cast<int32_t>(u);
    }
    wf[nw] = static_cast<int32_t>(units.size());
  }
  std::vector<int32_t> warp_of(units.size());
  for (int64_t w = 0; w < nw; ++w)
    for (int32_t u = wf[w]; u < wf[w + 1]; ++u) warp_of[u] = static_cast<int32_t>(w);
  size_t u = 0;
  while (u < units.size()) {
    size_t e = u;
    while (e < units.size() && units[e].zout == units[u].zout) ++e;  // block = units [u, e)
    const bool wide = static_cast<int64_t>(units[u].ldk) * static_cast<int64_t>(elem_bytes) > 32 * 16;
    std::vector<size_t> lasts;
    for (size_t v = u; v < e; ++v)
      if (wide || v + 1 == e || warp_of[v + 1] != warp_of[v]) lasts.push_back(v);
    if (lasts.size() == 1) {
      units[lasts[0]].flags = 1;
    } else {
      const int32_t g = static_cast<int32_t>(groups.size());
      groups.push_back(FarGroup{static_cast<int32_t>(ppos), static_cast<int32_t>(lasts.size()), units[u].zout,
                                units[u].k});
      for (size_t c = 0; c < lasts.size(); ++c) {
        FarUnit& L = units[lasts[c]];
        L.flags = 2;
        L.grp = g;
        L.zout = static_cast<int32_t>(ppos + static_cast<int64_t>(c) * L.ldk);
      }
      ppos += static_cast<int64_t>(lasts.size()) * units[u].ldk;
    }
    u = e;
  }
  nw_out = units.empty() ? 0 : nw;
  return wf;
}

// The stream plan of the single-vector apply, from the packing's units and segments: V^T units
// cut to tiles of at most ST_TILE bytes and dealt to the warps of ST_CTAS_PER_SM CTAs per SM; row
// items cut the same way into chunks, in segment order, dealt to as many CTAs.  Both by bytes
// plus the fixed cost of a tile, and to fewer warps when there would be less than 4 KB for each.
void cut_units(const std::vector<FarUnit>& in, const std::vector<FarGroup>& ing, size_t esz,
               std::vector<StUnit>& out) {
  const int E = 16 / static_cast<int>(esz);
  auto z_of = [&](const FarUnit& U) { return (U.flags & 3) == 2 ? ing[U.grp].zdst : U.zout; };  // of the block
  for (size_t q = 0; q < in.size(); ++q) {
    const FarUnit& U = in[q];
    const int32_t z = z_of(U);
    if (U.ldk > 32 * E) {  // more vectors than lanes: the block in strips of 32 vectors, row by row
      size_t e = q;
      while (e + 1 < in.size() && z_of(in[e + 1]) == z) ++e;
      for (int v = 0; v < U.ldk; v += 32 * E) {
        const int w = std::min(32 * E, U.ldk - v);
        for (size_t b = q; b <= e; ++b)
          for (int c = 0; c < in[b].nc; ++c)
            out.push_back(StUnit{in[b].voff + static_cast<int64_t>(c) * U.ldk + v, in[b].xc + c, z + v, -1,
                                 static_cast<int16_t>(w), 1, static_cast<int16_t>(std::max(0, std::min(w, U.k - v))), 0, 0,
                                 0});
      }
      q = e;
      continue;
    }
    int rows = static_cast<int>(ST_TILE / (U.ldk * (int64_t)esz));
    const int nv = U.ldk / E, round = ST_U * (32 / nv);  // rows of one round of tile_dot
    if (rows >= round) rows = rows / round * round;
    for (int a = 0; a < U.nc; a += rows) {
      const int e = std::min(U.nc, a + rows);
      out.push_back(StUnit{U.voff + static_cast<int64_t>(a) * U.ldk, U.xc + a, z, -1, static_cast<int16_t>(U.ldk),
                           static_cast<int16_t>(e - a), static_cast<int16_t>(U.k), 0, 0, 0});
    }
  }
}

// contiguous ranges of `n` things with prefix costs `cost` (n + 1) for `parts` workers
std::vector<int32_t> deal(const std::vector<double>& cost, int64_t parts) {
  const int64_t n = static_cast<int64_t>(cost.size()) - 1;
  std::vector<int32_t> f(parts + 1, 0);
  int64_t u = 0;
  for (int64_t w = 0; w <= parts; ++w) {
    const double target = cost.back() * static_cast<double>(w) / static_cast<double>(parts);
    while (u < n && cost[u] < target) ++u;
    f[w] = static_cast<int32_t>(u);
  }
  f[parts] = static_cast<int32_t>(n);
  return f;
}

// the warp ranges of a unit list; the last unit of a block in each warp writes the block (flags
// 1) or a partial of a group (flags 2, slots from *ppos)
std::vector<int32_t> deal_units(std::vector<StUnit>& units, size_t esz, size_t vsz, int64_t parts,
                                std::vector<FarGroup>& groups, int64_t& ppos) {
  std::vector<double> cost(units.size() + 1, 0.0);
  for (size_t u = 0; u < units.size(); ++u)
    cost[u + 1] = cost[u] + static_cast<double>(units[u].nc) * (units[u].ldk * esz + vsz) + 512.0;
  for (StUnit& U : units) {
    const int nv = U.ldk * static_cast<int>(esz) / 16;
    U.phases = static_cast<uint8_t>(32 / nv);
    U.magic = 65536 / nv + 1;  // lane / nv = (lane magic) >> 16 for lane < 32, nv <= 32
  }
  const std::vector<int32_t> wf = deal(cost, parts);
  std::vector<int32_t> warp_of(units.size());
  for (int64_t w = 0; w < parts; ++w)
    for (int32_t u = wf[w]; u < wf[w + 1]; ++u) warp_of[u] = static_cast<int32_t>(w);
  for (size_t u = 0; u < units.size();) {
    size_t e = u;
    while (e < units.size() && units[e].zout == units[u].zout) ++e;  // block = units [u, e)
    std::vector<size_t> lasts;
    for (size_t v = u; v < e; ++v)
      if (v + 1 == e || warp_of[v + 1] != warp_of[v]) lasts.push_back(v);
    if (lasts.size() == 1) {
      units[lasts[0]].flags = 1;
    } else {
      const int32_t g = static_cast<int32_t>(groups.size());
      groups.push_back(FarGroup{static_cast<int32_t>(ppos), static_cast<int32_t>(lasts.size()), units[u].zout,
                                units[u].k});
      const int32_t ldk = units[u].ldk;
      for (size_t c = 0; c < lasts.size(); ++c) {
        StUnit& L = units[lasts[c]];
        L.flags = 2;
        L.grp = g;
        L.zout = static_cast<int32_t>(ppos + static_cast<int64_t>(c) * ldk);
      }
      ppos += static_cast<int64_t>(lasts.size()) * ldk;
    }
    u = e;
  }
  return wf;
}
}  // namespace

void plan_stream(HMatrix& H, const std::vector<FarUnit>& units, const std::vector<FarUnit>& units_h,
                 const std::vector<FarGroup>& ugroups, const std::vector<int32_t>& seg, const std::vector<int64_t>& ip, const std::vector<int64_t>& hb,
                 const std::vector<int64_t>& nb, const std::vector<RowItem>& items, cudaStream_t s) {
  const size_t fsz = H.prec == Prec::F64 ? 8 : H.prec == Prec::MIXED ? 2 : 4, nsz = H.prec == Prec::F64 ? 8 : 4;
  const int nsm = num_sms(H.device);
  StreamPlan& S = H.st;
  // far_z
  std::vector<StUnit> zu, zh;
  cut_units(units, ugroups, fsz, zu);
  cut_units(units_h, ugroups, 2, zh);
  std::vector<FarGroup> groups;
  int64_t ppos = 0;
  auto bytes_of = [](const std::vector<StUnit>& us, size_t esz) {
    double b = 0.0;
    for (const StUnit& U : us) b += static_cast<double>(U.nc) * U.ldk * esz;
    return b;
  };
  const int64_t all = static_cast<int64_t>(nsm) * ST_CTAS_PER_SM * ST_WARPS;
  const int64_t nw = std::max<int64_t>(1, std::min<int64_t>(all, static_cast<int64_t>(bytes_of(zu, fsz) / 4096.0)));
  const std::vector<int32_t> wf = deal_units(zu, fsz, 8, nw, groups, ppos), wh = deal_units(zh, 2, 8, nw, groups, ppos);
  SPX_CHECK(ppos < (int64_t(1) << 31), "far-field partial slots exceed 2^31");
  auto check = [&](const std::vector<StUnit>& us, int64_t pool, size_t esz) {
    const int E = 16 / static_cast<int>(esz);
    for (const StUnit& U : us)
      SPX_CHECK(U.voff % E == 0 && U.ldk % E == 0 && U.nc >= 1 && U.ldk >= U.k && U.ldk <= 32 * E &&
                    static_cast<int64_t>(U.nc) * U.ldk * (int64_t)esz <= ST_TILE &&
                    U.voff + static_cast<int64_t>(U.nc) * U.ldk <= pool / (int64_t)esz && U.xc >= 0 &&
                    U.xc + static_cast<int64_t>(U.nc) <= H.Nb &&
                    U.zout + static_cast<int64_t>(U.k) <= (U.flags == 2 ? ppos : H.zlen),
                "stream plan: unit out of range");
  };
  check(zu, static_cast<int64_t>(H.far_f.n), fsz);
  check(zh, static_cast<int64_t>(H.far_h.n), 2);
  S.zpart_len = ppos;
  S.nzu = static_cast<int64_t>(zu.size());
  S.nzh = static_cast<int64_t>(zh.size());
  S.nwarps = nw;
  S.zu.upload(zu, s);
  S.zw.upload(wf, s);
  S.zh.upload(zh, s);
  S.zhw.upload(wh, s);
  S.zgroups.upload(groups, s);
  S.zcnt.alloc(std::max<size_t>(groups.size(), 1));
  S.zcnt.zero(s);
  // rows
  std::vector<StChunk> ch;
  std::vector<double> cost(1, 0.0);
  const int64_t nseg = static_cast<int64_t>(seg.size()) - 1;
  std::vector<int64_t> seg_c(nseg + 1, 0);
  for (int64_t g = 0; g < nseg; ++g) {
    const int nr = seg[g + 1] - seg[g];
    for (int64_t q = ip[g]; q < ip[g + 1]; ++q) {
      const int ty = q < hb[g] ? 0 : q < nb[g] ? 1 : 2;
      const size_t esz = ty == 0 ? fsz : ty == 1 ? 2 : nsz;
      const int E = 16 / static_cast<int>(esz), ld = (nr + E - 1) / E * E;
      const RowItem& I = items[q];
      int rows = static_cast<int>(ST_TILE / (ld * (int64_t)esz));
      const int round = ST_U * (32 / (ld / E));
      if (rows >= round) rows = rows / round * round;
      for (int a = 0; a < I.len; a += rows) {
        const int e = std::min(I.len, a + rows);
        ch.push_back(StChunk{I.off + static_cast<int64_t>(a) * ld, I.src + a, static_cast<uint16_t>(e - a),
                             static_cast<uint8_t>(ld), static_cast<uint8_t>(ty)});
        cost.push_back(cost.back() + static_cast<double>(e - a) * (ld * esz + 8.0) + 512.0);
      }
    }
    seg_c[g + 1] = static_cast<int64_t>(ch.size());
  }
  SPX_CHECK(ch.size() < (size_t(1) << 31), "too many row chunks");
  for (const StChunk& C : ch) {
    const int64_t esz = C.type == 0 ? (int64_t)fsz : C.type == 1 ? 2 : (int64_t)nsz;
    const int64_t pool = static_cast<int64_t>(C.type == 0 ? H.far_f.n : C.type == 1 ? H.far_h.n : H.near_f.n);
    SPX_CHECK(C.len >= 1 && C.off * esz % 16 == 0 && C.ld * esz % 16 == 0 &&
                  C.len * C.ld * esz <= ST_TILE && (C.off + static_cast<int64_t>(C.len) * C.ld) * esz <= pool &&
                  C.src >= 0 && C.src + static_cast<int64_t>(C.len) <= (C.type == 2 ? H.Nb : H.zlen),
              "stream plan: chunk out of range");
  }
  const int nctas = static_cast<int>(std::max<int64_t>(
      1, std::min<int64_t>(static_cast<int64_t>(nsm) * ST_CTAS_PER_SM, static_cast<int64_t>(cost.back() / (4096.0 * ST_WARPS)))));
  const std::vector<int32_t> cf = deal(cost, nctas);
  std::vector<StPortion> po;
  std::vector<int32_t> first(nctas + 1, 0);
  std::vector<std::vector<int32_t>> of_seg(nseg);  // portions of each segment
  int64_t g = 0;
  for (int c = 0; c < nctas; ++c) {
    int64_t a = cf[c];
    const int64_t e = cf[c + 1];
    // segments without chunks (no blocks on their rows) go to the CTA that reaches them
    while (g < nseg && (a < e || seg_c[g + 1] <= a)) {
      const int64_t b = std::min<int64_t>(seg_c[g + 1], e);
      if (b > a || seg_c[g + 1] == seg_c[g]) {
        of_seg[g].push_back(static_cast<int32_t>(po.size()));
        po.push_back(StPortion{seg[g], seg[g + 1] - seg[g], static_cast<int32_t>(a), static_cast<int32_t>(b), -1, 0});
      }
      a = b;
      if (seg_c[g + 1] <= a) ++g; else break;
    }
    first[c + 1] = static_cast<int32_t>(po.size());
  }
  SPX_CHECK(g == nseg, "row plan: not every segment was dealt");
  std::vector<int2> rg;
  int32_t slots = 0;
  for (int64_t q = 0; q < nseg; ++q) {
    if (of_seg[q].size() < 2) continue;
    const int32_t id = static_cast<int32_t>(rg.size());
    rg.push_back(make_int2(slots, static_cast<int>(of_seg[q].size())));
    for (int32_t p : of_seg[q]) {
      po[p].grp = id;
      po[p].slot = slots++;
    }
  }
  S.portions.upload(po, s);
  S.cta_first.upload(first, s);
  S.chunks.upload(ch, s);
  S.rgroups.upload(rg, s);
  S.rcnt.alloc(std::max<size_t>(rg.size(), 1));
  S.rcnt.zero(s);
  S.nslots = slots;
  S.nctas = nctas;
  S.ypart.alloc(std::max<int64_t>(slots, 1) * SEG_MAX);
  SPX_CUDA(cudaStreamSynchronize(s));  // the host vectors above back the uploads
}

namespace {
// FP32 columns kept by a recompressed block under the split packing: the trailing columns go
// to FP16 when their rounding (relative 2^-11 in U and in V) stays within a tenth of the
// block's error budget, sqrt(sum_{j>=c} 2 (sigma_j 2^-11)^2) <= 0.1 eps ||A||; rounded up to
// a multiple of 4 (the FP32 vector width); k (all FP32) without singular values.
int split_head(const std::vector<double>& sig, int k, double eps) {
  if (static_cast<int>(sig.size()) != k || k == 0) return k;
  double n2 = 0.0;
  for (double v : sig) n2 += v * v;
  const double bud = 0.1 * eps * std::sqrt(n2);
  const double u16 = std::ldexp(1.0, -11);
  double acc = 0.0;
  int c = k;
  for (int j = k - 1; j >= 0; --j) {
    acc += 2.0 * (sig[j] * u16) * (sig[j] * u16);
    if (std::sqrt(acc) > bud) break;
    c = j;
  }
  const int c4 = static_cast<int>(round_up(c, 4));
  return c4 >= k ? k : c4;
}

template <class TF, class TN>
void do_pack(HMatrix& H, cudaStream_t s, bool split = false) {
  constexpr int EF = 16 / static_cast<int>(sizeof(TF));
  constexpr int EN = 16 / static_cast<int>(sizeof(TN));
  constexpr int EH = 8;  // FP16 elements per 16 bytes
  // row segments: leaf clusters in permutation order, cut into pieces of <= SEG_MAX rows
  std::vector<int32_t> ls;
  for (const TreeNode& nd : H.tree.nodes)
    if (nd.leaf()) ls.push_back(nd.start);
  std::sort(ls.begin(), ls.end());
  ls.push_back(static_cast<int32_t>(H.Nb));
  std::vector<int32_t> seg;
  for (size_t l = 0; l + 1 < ls.size(); ++l) {
    const int32_t a = ls[l], n = ls[l + 1] - ls[l];
    const int32_t pieces = (n + SEG_MAX - 1) / SEG_MAX;
    for (int32_t p = 0; p < pieces; ++p) seg.push_back(a + static_cast<int32_t>((int64_t)n * p / pieces));
  }
  seg.push_back(static_cast<int32_t>(H.Nb));
  const int64_t nseg = static_cast<int64_t>(seg.size()) - 1;

  std::vector<PackJob> jf, jn, jh;
  std::vector<FarUnit> units, units_h;
  std::vector<std::vector<RowItem>> far_items(nseg), half_items(nseg), near_items(nseg);
  std::vector<double> scale;  // 1 / sigma of the FP16 columns of U (pack), sigma per z entry (apply)
  std::vector<double> zsc;
  int64_t fpos = 0, hpos = 0, npos = 0, zpos = 0, nf = 0, nn = 0;
  for (size_t bi = 0; bi < H.blocks.size(); ++bi) {
    const HBlock& b = H.blocks[bi];
    const int32_t m = b.re - b.rs, n = b.ce - b.cs;
    int64_t sg = std::upper_bound(seg.begin(), seg.end(), b.rs) - seg.begin() - 1;
    SPX_CHECK(sg >= 0 && seg[sg] == b.rs, "block rows do not start at a segment boundary");
    if (b.type == 1) {
      const int32_t k = b.rank;
      const int32_t kh = split ? split_head(H.sigma.empty() ? std::vector<double>() : H.sigma[bi], k,
                                            H.cfg.epsilon) : k;  // FP32 columns
      const int32_t kt = k - kh;                                 // FP16 columns
      const int32_t ldk = static_cast<int32_t>(round_up(std::max(kh, 1), EF));
      const int64_t pv = fpos;
      // V^T head: n rows of ldk (row c = V[0..kh-1, c]); units of at most ~16 KB of rows
      jf.push_back(PackJob{b.off_v, pv, n, kh, ldk, 1, n});
      fpos = pv + static_cast<int64_t>(n) * ldk;
      if (kh > 0) {
        const int32_t uc = std::max<int32_t>(8, static_cast<int32_t>(16384 / (static_cast<int64_t>(ldk) * sizeof(TF))));
        for (int32_t c0 = 0; c0 < n; c0 += uc)
          units.push_back(FarUnit{pv + static_cast<int64_t>(c0) * ldk, ldk, std::min(uc, n - c0), b.cs + c0, kh,
                                  static_cast<int32_t>(zpos), -1, 0, 0});
      }
      int64_t sgu = sg;
      for (; sgu < nseg && seg[sgu] < b.re; ++sgu) {
        const int32_t a = seg[sgu], nr = seg[sgu + 1] - seg[sgu];
        const int32_t ld = static_cast<int32_t>(round_up(nr, EF));
        jf.push_back(PackJob{b.off_u + (a - b.rs), fpos, kh, nr, ld, m, 1});
        far_items[sgu].push_back(RowItem{fpos, kh, static_cast<int32_t>(zpos)});
        fpos = round_up(fpos + (int64_t)kh * ld, EF);
      }
      for (int32_t q = 0; q < kh; ++q) zsc.push_back(1.0);
      if (kt > 0) {
        // tail: unit columns of U (scaled by 1 / sigma) and unit rows of V in FP16; z of the
        // tail is scaled back by sigma in the row kernel
        const std::vector<double>& sig = H.sigma[bi];
        const int64_t s0 = static_cast<int64_t>(scale.size());
        for (int32_t q = 0; q < kt; ++q) scale.push_back(1.0 / sig[kh + q]);
        const int32_t ldh = static_cast<int32_t>(round_up(kt, EH));
        const int64_t ph = hpos;
        jh.push_back(PackJob{b.off_v + static_cast<int64_t>(kh) * n, ph, n, kt, ldh, 1, n});
        hpos = ph + static_cast<int64_t>(n) * ldh;
        const int32_t uc = std::max<int32_t>(8, static_cast<int32_t>(16384 / (static_cast<int64_t>(ldh) * 2)));
        for (int32_t c0 = 0; c0 < n; c0 += uc)
          units_h.push_back(FarUnit{ph + static_cast<int64_t>(c0) * ldh, ldh, std::min(uc, n - c0), b.cs + c0, kt,
                                    static_cast<int32_t>(zpos + kh), -1, 0, 0});
        for (sgu = sg; sgu < nseg && seg[sgu] < b.re; ++sgu) {
          const int32_t a = seg[sgu], nr = seg[sgu + 1] - seg[sgu];
          const int32_t ld = static_cast<int32_t>(round_up(nr, EH));
          PackJob J{b.off_u + static_cast<int64_t>(kh) * m + (a - b.rs), hpos, kt, nr, ld, m, 1};
          J.qs = s0;
          jh.push_back(J);
          half_items[sgu].push_back(RowItem{hpos, kt, static_cast<int32_t>(zpos + kh)});
          hpos = round_up(hpos + (int64_t)kt * ld, EH);
        }
        for (int32_t q = 0; q < kt; ++q) zsc.push_back(sig[kh + q]);
      }
      zpos += k;
      ++nf;
    } else {
      for (; sg < nseg && seg[sg] < b.re; ++sg) {
        const int32_t a = seg[sg], nr = seg[sg + 1] - seg[sg];
        const int32_t ld = static_cast<int32_t>(round_up(nr, EN));
        jn.push_back(PackJob{b.off_u + (int64_t)(a - b.rs) * n, npos, n, nr, ld, 1, n});
        near_items[sg].push_back(RowItem{npos, n, b.cs});
        npos = round_up(npos + (int64_t)n * ld, EN);
      }
      ++nn;
    }
  }
  SPX_CHECK(zpos < (int64_t(1) << 31), "far-field rank sum exceeds 2^31");
  H.n_far = nf;
  H.n_near = nn;
  H.zlen = zpos;
  H.far_f.alloc(std::max<int64_t>(fpos, 1) * sizeof(TF));
  H.near_f.alloc(std::max<int64_t>(npos, 1) * sizeof(TN));
  H.far_h.alloc(hpos > 0 ? hpos * 2 : 0);
  H.bytes_far = fpos * (int64_t)sizeof(TF) + hpos * 2;
  H.bytes_near = npos * (int64_t)sizeof(TN);
  const bool bf = (H.prec == Prec::MIXED);
  if (sizeof(TF) == 8) run_pack_jobs<double>(jf, H.far_pool64.p, nullptr, H.far_f.p, s);
  else if (bf) run_pack_jobs<__nv_bfloat16>(jf, H.far_pool64.p, nullptr, H.far_f.p, s);
  else run_pack_jobs<float>(jf, H.far_pool64.p, nullptr, H.far_f.p, s);
  if (sizeof(TN) == 8) run_pack_jobs<double>(jn, H.near_pool64.p, nullptr, H.near_f.p, s);
  else run_pack_jobs<float>(jn, H.near_pool64.p, nullptr, H.near_f.p, s);
  if (!jh.empty()) {
    DevBuf<double> dsc;
    dsc.upload(scale, s);
    run_pack_jobs<__half>(jh, H.far_pool64.p, dsc.p, H.far_h.p, s);
  }

  const int nsm = num_sms(H.device);
  std::vector<FarGroup> groups;
  int64_t ppos = 0, nw = 0;
  std::vector<int32_t> wf = plan_units(units, sizeof(TF), nsm, nw, groups, ppos);
  SPX_CHECK(ppos < (int64_t(1) << 31), "far-field partial slots exceed 2^31");
  auto check_units = [&](const std::vector<FarUnit>& us, int64_t cap, int E) {
    for (const FarUnit& U : us)
      SPX_CHECK(U.voff % E == 0 && U.nc >= 1 && U.k >= 1 && U.ldk % E == 0 && U.ldk >= U.k &&
                    U.voff + static_cast<int64_t>(U.nc) * U.ldk <= cap && U.xc >= 0 &&
                    U.xc + static_cast<int64_t>(U.nc) <= H.Nb &&
                    ((U.flags & 3) != 2 || (U.grp >= 0 && U.grp < static_cast<int64_t>(groups.size()) &&
                                            U.zout + static_cast<int64_t>(U.k) <= ppos)),
                "far_z plan: unit out of range");
  };
  check_units(units, fpos, EF);
  H.zpart_len = ppos;
  H.nunits = static_cast<int64_t>(units.size());
  H.nwarps_z = nw;
  H.units.upload(units, s);
  H.warp_first.upload(wf, s);
  H.groups.upload(groups, s);
  H.gcnt.alloc(std::max<size_t>(groups.size(), 1));
  H.gcnt.zero(s);

  std::vector<int64_t> ip(nseg + 1, 0), nb(nseg, 0), hb(nseg, 0);
  std::vector<RowItem> items;
  for (int64_t g = 0; g < nseg; ++g) {
    items.insert(items.end(), far_items[g].begin(), far_items[g].end());
    hb[g] = static_cast<int64_t>(items.size());
    items.insert(items.end(), half_items[g].begin(), half_items[g].end());
    nb[g] = static_cast<int64_t>(items.size());
    items.insert(items.end(), near_items[g].begin(), near_items[g].end());
    ip[g + 1] = static_cast<int64_t>(items.size());
  }
  H.nseg = nseg;
  H.seg_start.upload(seg, s);
  H.item_ptr.upload(ip, s);
  H.near_begin.upload(nb, s);
  H.items.upload(items, s);
  if (hpos > 0) H.zscale.upload(zsc, s);
  else H.zscale.release();
  SPX_CUDA(cudaStreamSynchronize(s));
  plan_stream(H, units, units_h, groups, seg, ip, hb, nb, items, s);
}

// launch that may start while the kernel before it in the stream finishes (pdl_wait inside)
template <class... KArgs, class... Args>
void launch_dependent(void (*k)(KArgs...), unsigned grid, unsigned block, size_t dyn, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = dyn;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  SPX_CUDA(cudaLaunchKernelEx(&cfg, k, static_cast<KArgs>(args)...));
}

template <class TF, class TN, class TA, class TS>
void launch_apply(HMatrix& H, const TS* src, const int32_t* gidx, TS* dst, const TS* add, TS* yb, TA* xp, TA* z,
                  TA* zpart, cudaStream_t s) {
  const int64_t Nb = H.Nb;
  StreamPlan& S = H.st;
  k_hgather<TS, TA><<<grid_for(Nb, 256), 256, 0, s>>>(Nb, src, gidx, H.perm.p, xp);
  SPX_LAUNCH_CHECK();
  const unsigned ctas = static_cast<unsigned>(S.nctas), threads = ST_THREADS,
                 zctas = static_cast<unsigned>((S.nwarps + ST_WARPS - 1) / ST_WARPS);
  if (S.nzu > 0)
    launch_dependent(k_far_z<TF, TA>, zctas, threads, 0, s, S.zu.p, S.zw.p, static_cast<int>(S.nwarps),
                     reinterpret_cast<const TF*>(H.far_f.p), xp, z, zpart, S.zgroups.p, S.zcnt.p,
                     static_cast<const double*>(nullptr));
  if (S.nzh > 0)  // FP16 trailing columns of the split packing, scaled back by their singular values
    launch_dependent(k_far_z<__half, TA>, zctas, threads, 0, s, S.zh.p, S.zhw.p, static_cast<int>(S.nwarps),
                     reinterpret_cast<const __half*>(H.far_h.p), xp, z, zpart, S.zgroups.p, S.zcnt.p, H.zscale.p);
  launch_dependent(k_rows<TF, TN, TA, TS>, ctas, threads, 0, s, S.portions.p, S.cta_first.p, S.chunks.p,
                   reinterpret_cast<const TF*>(H.far_f.p), reinterpret_cast<const TN*>(H.near_f.p),
                   S.nzh > 0 ? reinterpret_cast<const __half*>(H.far_h.p) : static_cast<const __half*>(nullptr), z, xp, H.diag_perm.p, H.perm.p, gidx, dst, add, yb,
                   S.rgroups.p, S.rcnt.p, reinterpret_cast<TA*>(S.ypart.p));
}

template <class TF, class TN, class TA, class TS>
void do_apply(HMatrix& H, const TS* src, const int32_t* gidx, TS* dst, const TS* add, TS* yb, cudaStream_t s) {
  const size_t xb = H.Nb * sizeof(TA), zb = std::max<int64_t>(H.zlen, 1) * sizeof(TA),
               pb = std::max<int64_t>(H.st.zpart_len, 1) * sizeof(TA);
  if (H.xperm.n < xb) H.xperm.alloc(xb);
  if (H.z.n < zb) H.z.alloc(zb);
  if (H.zpart.n < pb) H.zpart.alloc(pb);
  launch_apply<TF, TN, TA, TS>(H, src, gidx, dst, add, yb, reinterpret_cast<TA*>(H.xperm.p),
                               reinterpret_cast<TA*>(H.z.p), reinterpret_cast<TA*>(H.zpart.p), s);
}
}  // namespace

void HMatrix::pack(Prec p, cudaStream_t s) {
  if (p == Prec::SPLIT && !recompressed) recompress(s);  // the split needs SVD-ordered columns
  tr.reset();
  prec = p;
  switch (p) {
    case Prec::F64: do_pack<double, double>(*this, s); break;
    case Prec::F32: do_pack<float, float>(*this, s); break;
    case Prec::MIXED: do_pack<__nv_bfloat16, float>(*this, s); break;
    case Prec::SPLIT: do_pack<float, float>(*this, s, true); break;
  }
  packed = true;
}

template <class T>
void HMatrix::apply_gather(const T* src, const int32_t* gidx, T* dst, const T* add, T* yb, cudaStream_t s) {
  SPX_CHECK(packed, "H-matrix is not packed");
  // FP64 vectors accumulate in FP64 whatever the factor storage; FP32 vectors in FP32
  if (sizeof(T) == sizeof(double)) {
    switch (prec) {
      case Prec::F64: do_apply<double, double, double, T>(*this, src, gidx, dst, add, yb, s); break;
      case Prec::F32:
      case Prec::SPLIT: do_apply<float, float, double, T>(*this, src, gidx, dst, add, yb, s); break;
      case Prec::MIXED: do_apply<__nv_bfloat16, float, double, T>(*this, src, gidx, dst, add, yb, s); break;
    }
  } else {
    switch (prec) {
      case Prec::F64: do_apply<double, double, float, T>(*this, src, gidx, dst, add, yb, s); break;
      case Prec::F32:
      case Prec::SPLIT: do_apply<float, float, float, T>(*this, src, gidx, dst, add, yb, s); break;
      case Prec::MIXED: do_apply<__nv_bfloat16, float, float, T>(*this, src, gidx, dst, add, yb, s); break;
    }
  }
}
template void HMatrix::apply_gather<double>(const double*, const int32_t*, double*, const double*, double*, cudaStream_t);
template void HMatrix::apply_gather<float>(const float*, const int32_t*, float*, const float*, float*, cudaStream_t);

void HMatrix::apply_f64(const double* x, double* y, cudaStream_t s) {
  apply_gather<double>(x, nullptr, y, nullptr, nullptr, s);
}

int64_t HMatrix::device_bytes() const {
  return static_cast<int64_t>(far_f.bytes() + near_f.bytes() + units.bytes() + warp_first.bytes() + groups.bytes() +
                              gcnt.bytes() + seg_start.bytes() + item_ptr.bytes() + near_begin.bytes() +
                              items.bytes() + z.bytes() + zpart.bytes() + xperm.bytes() + diag_perm.bytes() +
                              perm.bytes() + far_h.bytes() + zscale.bytes() + st.bytes());
}

}  // namespace spx

// ------------------------------------------------------------------ apply without allocation
// spx_hmat_apply_noalloc runs the same three kernels as spx_hmat_apply, but its scratch
// (x in permuted order, the far-field z vectors and the partial sums of long rows) lives in
// this fixed device array instead of buffers allocated on first use.  Every device that
// loads the library holds the array until the process exits.  In host code the symbol is
// only a stand-in: the device address comes from cudaGetSymbolAddress, looked up once per
// device.
namespace spx {

constexpr size_t kNoAllocScratchBytes = size_t(32) << 20;  // 32 MiB
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
std::atomic<int64_t> g_noalloc_cap{0};  // test cap on the accepted scratch size (0: none)

namespace {

void* noalloc_scratch_address() {
  static std::mutex mu;
  static std::vector<void*> addr;
  int dev = 0;
  SPX_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (static_cast<size_t>(dev) >= addr.size()) addr.resize(dev + 1, nullptr);
  if (!addr[dev]) {
    void* p = nullptr;
    SPX_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    addr[dev] = p;
  }
  return addr[dev];
}

template <class TF, class TN, class TA>
void apply_noalloc_impl(HMatrix& H, const double* x, double* y, cudaStream_t s) {
  const int64_t Nb = H.Nb;
  const size_t xbytes = ((static_cast<size_t>(Nb) * sizeof(TA) + 255) / 256) * 256;
  const size_t zbytes = ((static_cast<size_t>(std::max<int64_t>(H.zlen, 1)) * sizeof(TA) + 255) / 256) * 256;
  const size_t pbytes = static_cast<size_t>(std::max<int64_t>(H.st.zpart_len, 1)) * sizeof(TA);
  const int64_t cap = g_noalloc_cap.load();
  const size_t limit = cap > 0 ? std::min(kNoAllocScratchBytes, static_cast<size_t>(cap)) : kNoAllocScratchBytes;
  if (xbytes + zbytes + pbytes > limit)
    throw Error(ERR_INVALID, "H-matrix too large for the " + std::to_string(limit) +
                             "-byte static scratch of spx_hmat_apply_noalloc (needs " +
                             std::to_string(xbytes + zbytes + pbytes) + " bytes); use spx_hmat_apply");
  unsigned char* base = static_cast<unsigned char*>(noalloc_scratch_address());
  launch_apply<TF, TN, TA, double>(H, x, nullptr, y, nullptr, nullptr, reinterpret_cast<TA*>(base),
                                   reinterpret_cast<TA*>(base + xbytes), reinterpret_cast<TA*>(base + xbytes + zbytes),
                                   s);
}

}  // namespace

void hmat_apply_noalloc(HMatrix& H, const double* x, double* y, cudaStream_t s) {
  SPX_CHECK(H.packed, "H-matrix is not packed");
  switch (H.prec) {
    case Prec::F64: apply_noalloc_impl<double, double, double>(H, x, y, s); break;
    case Prec::F32:
    case Prec::SPLIT: apply_noalloc_impl<float, float, double>(H, x, y, s); break;
    case Prec::MIXED: apply_noalloc_impl<__nv_bfloat16, float, double>(H, x, y, s); break;
  }
}

}  // namespace spx
