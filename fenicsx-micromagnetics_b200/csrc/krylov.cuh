// Pieces of the persistent Krylov kernels: the group of CTAs that runs one solve, its barrier
// and its sums.
#pragma once

#include "spx_internal.cuh"

namespace spx {

// The CTAs of a solve: one CTA (TEAM_CTA), one cluster (TEAM_CLUSTER) or the whole cooperative
// grid, in a form with as few barriers as there can be (TEAM_GRID) or with as few bytes
// (TEAM_GRID_LARGE).  A barrier costs 1.3 us over the grid, so small systems run on one CTA or
// one cluster, whose barriers are in hardware.
enum : int { TEAM_CTA = 0, TEAM_CLUSTER = 1, TEAM_GRID = 2, TEAM_GRID_LARGE = 3 };
constexpr int TEAM_MAX_CLUSTER = 8;  // portable cluster size

struct TeamShared {
  double red[2][64];                    // per-warp partials of the two sums, two slots
  double cta[2][2 * TEAM_MAX_CLUSTER];  // per-CTA partials (cluster)
  double tot[2];
  int ok;
};

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 32-bit address of a shared-memory location of this CTA in CTA `rank` of the cluster
__device__ __forceinline__ unsigned cluster_addr(unsigned local, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
// store to the same shared-memory location of CTA `rank` of the cluster
__device__ __forceinline__ void cluster_store(double* local, unsigned rank, double v) {
  const unsigned r = cluster_addr(static_cast<unsigned>(__cvta_generic_to_shared(local)), rank);
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
}

// load by such an address (by a CTA-local one when the team is one CTA); volatile: the same
// location is written by its owner between two barriers
template <int TEAM>
__device__ __forceinline__ float team_load(unsigned a, float) {
  float v;
  if constexpr (TEAM == TEAM_CLUSTER)
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  else
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
template <int TEAM>
__device__ __forceinline__ double team_load(unsigned a, double) {
  double v;
  if constexpr (TEAM == TEAM_CLUSTER)
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  else
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}

// Barrier over the team; false when a bounded grid wait gave up.
template <int TEAM>
__device__ __forceinline__ bool team_barrier(unsigned int* bar, int* err) {
  if constexpr (TEAM == TEAM_CTA) {
    __syncthreads();
    return true;
  } else if constexpr (TEAM == TEAM_CLUSTER) {
    cluster_sync_all();
    return true;
  } else {
    return grid_barrier(bar, nullptr, gridDim.x, err);
  }
}

// Barrier with two sums over the team's threads, the same bits in every thread.  `flip`
// alternates the slots of the partials: a slot is written again only after the barrier that
// follows every thread's last read of it.  part: 4 x gridDim.x doubles (grid).
template <int TEAM>
__device__ __forceinline__ bool team_sum(TeamShared& S, double* part_base, unsigned int* bar, int* err, int& flip,
                                         double& a, double& b) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  a = warp_sum(a);
  b = warp_sum(b);
  double* red = S.red[flip];
  if (lane == 0) {
    red[2 * wid] = a;
    red[2 * wid + 1] = b;
  }
  __syncthreads();
  const int f = flip;
  flip ^= 1;
  if constexpr (TEAM == TEAM_CTA) {
    a = warp_sum(lane < nw ? red[2 * lane] : 0.0);
    b = warp_sum(lane < nw ? red[2 * lane + 1] : 0.0);
    return true;
  } else if constexpr (TEAM == TEAM_CLUSTER) {
    const int nb = gridDim.x;  // one cluster
    if (wid == 0) {
      const double u = warp_sum(lane < nw ? red[2 * lane] : 0.0);
      const double v = warp_sum(lane < nw ? red[2 * lane + 1] : 0.0);
      if (lane < nb) {
        cluster_store(&S.cta[f][2 * blockIdx.x], lane, u);
        cluster_store(&S.cta[f][2 * blockIdx.x + 1], lane, v);
      }
    }
    cluster_sync_all();
    a = warp_sum(lane < nb ? S.cta[f][2 * lane] : 0.0);
    b = warp_sum(lane < nb ? S.cta[f][2 * lane + 1] : 0.0);
    return true;
  } else {
    const int nb = gridDim.x;
    if (wid == 0) {
      double u = warp_sum(lane < nw ? red[2 * lane] : 0.0);
      double v = warp_sum(lane < nw ? red[2 * lane + 1] : 0.0);
      double* part = part_base + static_cast<int64_t>(f) * 2 * nb;
      if (lane == 0) {
        part[2 * blockIdx.x] = u;
        part[2 * blockIdx.x + 1] = v;
        S.ok = grid_arrive_wait(bar, nb, err) ? 1 : 0;
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
    __syncthreads();
    a = S.tot[0];
    b = S.tot[1];
    return S.ok != 0;
  }
}

}  // namespace spx
