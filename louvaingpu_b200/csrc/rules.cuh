// Device rules of a pass shared by the level kernels and the small-graph
// kernel: candidate order, moves, commit, modularity terms, row sums.
#pragma once
#include <climits>

#include "louvain.cuh"

namespace lvg {

constexpr int kNone = INT_MAX;   // no candidate community

__device__ __forceinline__ void delta_clear(Delta& d) {
  d.tot = 0.0; d.in = 0.0; d.size = 0; d.out = 0; d.iw_out = 0.0;
}

// Commit of one community's pass deltas (communitySetKernel,
// OneLevelKernel.cu:93-107): tot/in/size move by the deltas, and a vertex
// that left its singleton community takes its degree and weight out of it.
__device__ __forceinline__ void delta_commit(Delta& d, double kc, double& tot, double& in, int32_t& size) {
  double t = tot, x = in;
  if (d.out) { t = __dsub_rn(t, kc); x = __dsub_rn(x, d.iw_out); }
  tot = __dadd_rn(t, d.tot);
  in = __dadd_rn(x, d.in);
  size += d.size - d.out;
  delta_clear(d);
}

// Segmented inclusive warp sum over contiguous runs of equal `seg`.
template <typename K>
__device__ __forceinline__ double seg_warp_sum(double v, K seg) {
  const unsigned full = 0xffffffffu;
  int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    double u = __shfl_up_sync(full, v, o);
    K t = __shfl_up_sync(full, seg, o);
    if (lane >= o && t == seg) v = __dadd_rn(v, u);
  }
  return v;
}

template <typename K>
__device__ __forceinline__ bool seg_warp_last(K seg, bool valid) {
  const unsigned full = 0xffffffffu;
  int lane = threadIdx.x & 31;
  K nx = __shfl_down_sync(full, seg, 1);
  bool nvalid = __shfl_down_sync(full, valid, 1);
  return valid && (lane == 31 || !nvalid || nx != seg);
}

// Runs of equal `seg` in a warp (lanes hold consecutive list entries): the
// lane's distance from its run's first lane, and whether it is the run's last.
// Two votes and a shuffle, where a scan that shuffles `seg` along needs one a
// step: the shuffles are what bounds the scans below.
__device__ __forceinline__ int run_depth(int32_t seg, bool& last) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int32_t before = __shfl_up_sync(full, seg, 1);
  const unsigned heads = __ballot_sync(full, lane == 0 || before != seg);
  last = lane == 31 || ((heads >> (lane + 1)) & 1u);
  return lane - (31 - __clz(heads & (0xffffffffu >> (31 - lane))));
}

// Inclusive sum over the lanes of v's run up to this one, from run_depth.
__device__ __forceinline__ double run_sum(double v, int depth) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double u = __shfl_up_sync(0xffffffffu, v, o);
    if (o <= depth) v = __dadd_rn(v, u);
  }
  return v;
}

__device__ __forceinline__ uint64_t edge_hash(uint32_t u, uint32_t v, uint32_t wb, uint64_t key) {
  return mix64(mix64((((uint64_t)u << 32) | v) ^ key) + (uint64_t)wb * 0x9E3779B97F4A7C15ull + key);
}

// Candidate order: higher gain first, then lower community id
// (OneLevelKernel.cu:330,358).  Only strictly positive gains are candidates.
__device__ __forceinline__ bool better(double g2, int32_t c2, double g1, int32_t c1) {
  return g2 > g1 || (g2 == g1 && c2 < c1);
}

// Halves of a positive double, whose bits order as its value does.
__device__ __forceinline__ uint32_t gain_hi(double x) { return (uint32_t)__double2hiint(x); }
__device__ __forceinline__ uint32_t gain_lo(double x) { return (uint32_t)__double2loint(x); }

// remove/insert (OneLevelKernel.cu:52-78) of a vertex of degree ki moving
// with weight iw from community own to best.  SINGLETON: own holds only this
// vertex, so its side is two plain stores the commit applies.
template <bool SINGLETON>
__device__ __forceinline__ void move_deltas(Delta* d, int32_t own, int32_t best, double ki, double iw) {
  if (SINGLETON) {
    d[own].out = 1;
    d[own].iw_out = iw;
  } else {
    atomicAdd(&d[own].tot, -ki);
    atomicAdd(&d[own].in, -iw);
    atomicAdd(&d[own].size, -1);
  }
  atomicAdd(&d[best].tot, ki);
  atomicAdd(&d[best].in, iw);
  atomicAdd(&d[best].size, 1);
}

// term_c = in_c/m - (tot_c/2m)^2 (OneLevelKernel.cu:447-448), zero when m <= 0.
__device__ __forceinline__ double q_term(double in, double tot, double m, double twom) {
  if (!(m > 0.0)) return 0.0;
  double a = __ddiv_rn(in, m);
  double b = __ddiv_rn(tot, twom);
  return __dsub_rn(a, __dmul_rn(b, b));
}

__device__ __forceinline__ bool entry_ok(int32_t u, int32_t v, float x, int32_t V) {
  return u >= 0 && u < V && v >= 0 && v < V && x >= 0.0f && !isinf(x);   // as list_facts_kernel
}

}  // namespace lvg
