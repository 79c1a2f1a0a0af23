// Small graphs: all levels of a dendrogram in one launch.
//
// The level kernels take about 70 launches and 17 host reads of sizes a
// level, some 0.7 ms however small the level is.  Here a thread-block cluster
// (one block to sixteen) runs the whole level loop of one graph: the phases of
// a level are separated by cluster barriers instead of launches, every
// decision of the loop (the ΔQ test, the level break, sizes) is taken by all
// threads from the same values, and the host reads one result at the end.  In
// a batch each graph has its own cluster, so the graphs' levels need not wait
// for one another.
//
// A level's list is strictly sorted by (src, dst) and symmetric, so a row is a
// contiguous range of the list and the merged CSR entry of (u, v, w) is
// (u, v, 2w); no CSR is written.  The rules are the level kernels' (rules.cuh):
//   build    row starts, degrees and self loops from one pass over the list,
//            m and every Q on the fixed tree
//   pass 1   singletons: the best candidate of a row is an argmax over its
//            entries (segmented warp argmax, then shared-memory max / min)
//   pass 2+  tiles of consecutive rows hashed as (row, community) pairs in
//            shared memory: packed 64-bit slots when the weights are integral,
//            key + FP64 sum otherwise
//   renumber by smallest member; coarse keys (cu << b | cv) sorted by a stable
//            LSD radix sort across the cluster, runs summed in FP64
// A list that is not sorted and symmetric, a row longer than a tile, or more
// levels or passes than the tables hold end the launch with the level left
// open; the caller goes on with the level kernels from the same list.
#include <algorithm>
#include <cooperative_groups.h>
#include <mutex>

#include "prims.cuh"
#include "rules.cuh"
#include "small.cuh"

namespace lvg {
namespace {

namespace cg = cooperative_groups;

constexpr int kTileInt = 4096;             // entries of a tile, packed slots
constexpr int kSlots = 2 * kTileInt;       // 64 KB of slots, at most half full
constexpr int kTileF64 = kTileInt / 2;     // key + sum take two slots
constexpr int kTileRows = 1024;            // rows of a tile (10 bits of a packed key)
constexpr int kCommBits = 16;              // community bits of a packed key
constexpr int kDigits = 256;
constexpr unsigned long long kEmpty = ~0ull;
static_assert(kSmallMaxV <= (1 << kCommBits), "packed keys hold 16-bit communities");
static_assert(kTileRows <= (1 << 10) && kTileInt < (1 << 14), "packed key or claimed slot too wide");

enum : uint32_t { fNotInt = 1u, fUnfit = 2u, fBad = 4u, fUnsorted = 8u };

// Shared control words of a job (device memory).
struct Ctl {
  uint32_t flags, flags2, check, loops;
  unsigned long long sums[2];
  uint32_t count[2][16];
};

struct Work {
  Ctl* ctl;
  double *k, *kfrac, *tot, *in, *qpart, *mpart;
  Delta* delta;
  int32_t *roff, *comm, *next, *cand, *size, *minidx, *newid, *part;
  float* loopw;
  int32_t* hasl;
  uint32_t *key[2], *ghist;
  float* val[2];
  double* wsum;
};

__host__ __device__ inline size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

__host__ __device__ inline size_t carve(char* base, int64_t V, int64_t E, Work& W) {
  size_t o = 0;
  auto take = [&](size_t bytes) {
    char* p = base + o;
    o += up256(bytes);
    return p;
  };
  W.ctl = (Ctl*)take(sizeof(Ctl));
  W.k = (double*)take(8 * V);
  W.kfrac = (double*)take(8 * V);
  W.tot = (double*)take(8 * V);
  W.in = (double*)take(8 * V);
  W.qpart = (double*)take(8 * (V / kGroup + 1));
  W.mpart = (double*)take(8 * (E / kGroup + V / kGroup + 2));
  W.delta = (Delta*)take(sizeof(Delta) * V);
  W.roff = (int32_t*)take(4 * (V + 1));
  W.comm = (int32_t*)take(4 * V);
  W.next = (int32_t*)take(4 * V);
  W.cand = (int32_t*)take(4 * V);
  W.size = (int32_t*)take(4 * V);
  W.minidx = (int32_t*)take(4 * V);
  W.newid = (int32_t*)take(4 * V);
  W.part = (int32_t*)take(4 * V);
  W.loopw = (float*)take(4 * V);
  W.hasl = (int32_t*)take(4 * V);
  W.key[0] = (uint32_t*)take(4 * E);
  W.key[1] = (uint32_t*)take(4 * E);
  W.val[0] = (float*)take(4 * E);
  W.val[1] = (float*)take(4 * E);
  W.wsum = (double*)take(8 * E);
  W.ghist = (uint32_t*)take(4 * kDigits * 16);
  return o;
}

__host__ __device__ inline void list_of(char* lists, int64_t E, int buf, int32_t** src, int32_t** dst, float** w) {
  char* p = lists + (size_t)buf * 3 * up256(4 * E);
  *src = (int32_t*)p;
  *dst = (int32_t*)(p + up256(4 * E));
  *w = (float*)(p + 2 * up256(4 * E));
}

template <int NT>
struct Smem {
  union {
    unsigned long long slot[kSlots];
    uint32_t wc[NT / 32][kDigits + 1];
  } u;
  unsigned long long bestg[kTileRows];
  double bestw[kTileRows];
  double kf[kTileRows];
  int32_t bestc[kTileRows];
  int32_t own[kTileRows];
  int32_t nseg[kTileRows];   // distinct candidate communities; bit 30: own community seen
  uint16_t claimed[kTileInt];
  uint32_t hist[kDigits];
  uint32_t dbase[kDigits];
  double ws[NT / 256][8];
  double bcast;
  uint32_t wtot[NT / 32];
  int32_t nclaimed;
};

// ------------------------------------------------------------------ the cluster
template <int NT>
struct Team {
  int K, rank, tid;
  __device__ int gt() const { return rank * NT + tid; }
  __device__ int stride() const { return K * NT; }
  // Barrier of the job's threads; global writes before it are seen after it.
  __device__ void sync() const {
    if (K == 1) {
      __syncthreads();
    } else {
      __threadfence();
      cg::this_cluster().sync();
    }
  }
};

template <int NT>
__device__ __forceinline__ uint32_t block_excl(uint32_t v, uint32_t* wtot, uint32_t* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t inc = warp_inclusive_scan(v);
  if (lane == 31) wtot[w] = inc;
  __syncthreads();
  if (w == 0) {
    uint32_t x = lane < NT / 32 ? wtot[lane] : 0u;
    x = warp_inclusive_scan(x);
    if (lane < NT / 32) wtot[lane] = x;
  }
  __syncthreads();
  const uint32_t base = w > 0 ? wtot[w - 1] : 0u;
  *total = wtot[NT / 32 - 1];
  __syncthreads();
  return base + inc - v;
}

// block_tree256 of each 256-thread quarter; the result in its first thread.
template <int NT>
__device__ __forceinline__ double quarter_tree(double s, Smem<NT>& S) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = (threadIdx.x & 255) >> 5, q = threadIdx.x >> 8;
  for (int o = 16; o >= 1; o >>= 1) s = __dadd_rn(s, __shfl_down_sync(full, s, o));
  if (lane == 0) S.ws[q][w] = s;
  __syncthreads();
  double r = 0.0;
  if (w == 0) {
    double v = lane < 8 ? S.ws[q][lane] : 0.0;
    for (int o = 16; o >= 1; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(full, v, o));
    r = v;
  }
  __syncthreads();
  return r;
}

// Group partials of the fixed-tree sum of val(i), i < n (groups of 2048, a
// quarter block each); val is called once per index.
template <int NT, typename F>
__device__ __forceinline__ void group_partials(const Team<NT>& T, Smem<NT>& S, int64_t n, double* partials, F val) {
  const int64_t ng = max((int64_t)1, (n + kGroup - 1) / kGroup);
  const int nq = NT / 256, q = T.tid >> 8, t = T.tid & 255;
  for (int64_t g0 = (int64_t)T.rank * nq; g0 < ng; g0 += (int64_t)T.K * nq) {
    const int64_t g = g0 + q;
    double s = 0.0;
    if (g < ng) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int64_t i = g * kGroup + j * 256 + t;
        if (i < n) s = __dadd_rn(s, val(i));
      }
    }
    const double r = quarter_tree<NT>(s, S);
    if (t == 0 && g < ng) partials[g] = r;
  }
}

// Sum of the partials of n values, in every thread (at most 2048 partials).
template <int NT>
__device__ __forceinline__ double finish_sum(Smem<NT>& S, const double* partials, int64_t n) {
  const int64_t np = max((int64_t)1, (n + kGroup - 1) / kGroup);
  double s = 0.0;
  if (threadIdx.x < 256) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int64_t i = j * 256 + (int)threadIdx.x;
      if (i < np) s = __dadd_rn(s, partials[i]);
    }
  }
  const double r = quarter_tree<NT>(s, S);
  if (threadIdx.x == 0) S.bcast = r;
  __syncthreads();
  const double x = S.bcast;
  __syncthreads();
  return x;
}

// First v in [0, V] with roff[v] >= x.
__device__ __forceinline__ int32_t row_at(const int32_t* roff, int32_t V, int64_t x) {
  int32_t lo = 0, hi = V;
  while (lo < hi) {
    const int32_t mid = (lo + hi) >> 1;
    if (roff[mid] >= x) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// The decision for one vertex (apply_decision_kl of the level kernels).
template <bool SINGLETON>
__device__ __forceinline__ void decide(const Work& W, int32_t i, int32_t own, int32_t bc, double bw, int32_t nseg) {
  const int32_t raw = bc == kNone ? own : bc;
  const int32_t so = SINGLETON ? 1 : W.size[own], sb = SINGLETON ? 1 : W.size[raw];
  int32_t best = raw;
  if (so == 1 && sb == 1 && raw > own) best = own;
  W.next[i] = best;
  W.cand[i] = (so == 1 && nseg == 1 && raw != own && own < raw) ? raw : -1;
  if (best != own) move_deltas<SINGLETON>(W.delta, own, best, W.k[i], __dadd_rn(bw, (double)W.loopw[i]));
}

// Rows [v0, v0 + return value) of the next tile: at most `cap` entries and
// kTileRows rows.  Uniform over the block.
template <int NT>
__device__ __forceinline__ int tile_rows(const int32_t* roff, int32_t v0, int32_t vend, int cap) {
  const int32_t base = roff[v0];
  int nv = 0;
  for (int x = threadIdx.x; x < kTileRows; x += NT) {
    const int32_t v = v0 + 1 + x;
    nv += __syncthreads_count(v <= vend && roff[v] - base <= cap);
  }
  return nv;
}

struct List {
  const int32_t* src;
  const int32_t* dst;
  const float* w;
};

__device__ __forceinline__ double merged_w(float w) { return (double)__double2float_rn(__dadd_rn((double)w, (double)w)); }

// First pass of a level: every neighbour is its own candidate.
template <int NT>
__device__ void moves_first(const Team<NT>& T, Smem<NT>& S, const Work& W, const List& L, int32_t v, int32_t vend) {
  constexpr int kItems = kTileInt / NT;
  const unsigned full = 0xffffffffu;
  const int lane = T.tid & 31;
  while (v < vend) {
    const int nv = tile_rows<NT>(W.roff, v, vend, kTileInt);
    if (nv == 0) return;   // cannot happen: rows longer than a tile leave the level open
    const int32_t base = W.roff[v];
    const int n = W.roff[v + nv] - base;
    if (n > 0) {
      for (int j = T.tid; j < nv; j += NT) {
        S.kf[j] = W.kfrac[v + j];
        S.bestg[j] = 0ull;
        S.bestc[j] = kNone;
      }
      int jj[kItems], cc[kItems];
      double gg[kItems], wd[kItems];
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        const int x = q * NT + T.tid;
        jj[q] = -1;
        cc[q] = 0;
        wd[q] = 0.0;
        if (x < n) {
          jj[q] = L.src[base + x] - v;
          cc[q] = L.dst[base + x];
          wd[q] = merged_w(L.w[base + x]);
        }
      }
#pragma unroll
      for (int q = 0; q < kItems; ++q) gg[q] = jj[q] >= 0 ? W.k[cc[q]] : 0.0;   // singleton tot = k
      __syncthreads();
      unsigned last = 0;
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        const int j = jj[q];
        double g = 0.0, w = wd[q];
        int32_t c = kNone;
        if (j >= 0 && cc[q] != v + j && w != 0.0) {                        // OneLevelKernel.cu:303
          const double t = __dsub_rn(w, __dmul_rn(gg[q], S.kf[j]));        // OneLevelKernel.cu:307-313
          if (t > 0.0) { g = t; c = cc[q]; }
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {   // best candidate of the lane's row piece so far
          const double g2 = __shfl_up_sync(full, g, o), w2 = __shfl_up_sync(full, w, o);
          const int32_t c2 = __shfl_up_sync(full, c, o), j2 = __shfl_up_sync(full, j, o);
          if (lane >= o && j2 == j && better(g2, c2, g, c)) { g = g2; c = c2; w = w2; }
        }
        const int32_t jn = __shfl_down_sync(full, j, 1);
        if (j >= 0 && c != kNone && (lane == 31 || jn != j)) {
          last |= 1u << q;
          atomicMax(&S.bestg[j], (unsigned long long)__double_as_longlong(g));
        }
        gg[q] = g;
        cc[q] = c;
        wd[q] = w;
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q)
        if ((last >> q) & 1u) {
          if ((unsigned long long)__double_as_longlong(gg[q]) == S.bestg[jj[q]]) atomicMin(&S.bestc[jj[q]], cc[q]);
          else last &= ~(1u << q);
        }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q)
        if (((last >> q) & 1u) && cc[q] == S.bestc[jj[q]]) S.bestw[jj[q]] = wd[q];
      __syncthreads();
      for (int j = T.tid; j < nv; j += NT) {
        const int32_t i = v + j, len = W.roff[i + 1] - W.roff[i];
        const int32_t c = S.bestc[j];
        // distinct candidates: one per neighbour, and the own community with a self loop
        if (len > 0) decide<true>(W, i, i, c, c == kNone ? 0.0 : S.bestw[j], len);
      }
      __syncthreads();
    }
    v += nv;
  }
}

// (row, community) tables.  Packed: row << 16 | community in the high half,
// integer sum in the low half; all ones when empty.
template <bool INT>
struct Table;

template <>
struct Table<true> {
  static constexpr int kTile = kTileInt;
  static __device__ __forceinline__ uint32_t hash(uint32_t key) {
    return (uint32_t)(((unsigned long long)key * 0x9E3779B97F4A7C15ull) >> (64 - 13));
  }
  static __device__ __forceinline__ void insert(unsigned long long* slot, int32_t* ncl, uint16_t* claimed, int j,
                                                int32_t c, double w) {
    const uint32_t key = ((uint32_t)j << kCommBits) | (uint32_t)c, wi = (uint32_t)w;
    uint32_t h = hash(key);
    for (int p = 0; p < kSlots; ++p) {   // at most half the slots are ever taken
      const unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(&slot[h]);
      if ((uint32_t)(cur >> 32) == key) { atomicAdd(&slot[h], (unsigned long long)wi); return; }
      if (cur == kEmpty) {
        const unsigned long long prev = atomicCAS(&slot[h], kEmpty, ((unsigned long long)key << 32) | wi);
        if (prev == kEmpty) { claimed[atomicAdd(ncl, 1)] = (uint16_t)h; return; }
        if ((uint32_t)(prev >> 32) == key) { atomicAdd(&slot[h], (unsigned long long)wi); return; }
      }
      h = (h + 1) & (kSlots - 1);
    }
  }
  static __device__ __forceinline__ void get(const unsigned long long* slot, int s, int& j, int32_t& c, double& w) {
    const unsigned long long x = slot[s];
    const uint32_t key = (uint32_t)(x >> 32);
    j = (int)(key >> kCommBits);
    c = (int32_t)(key & ((1u << kCommBits) - 1u));
    w = (double)(uint32_t)x;
  }
  static __device__ __forceinline__ void clear(unsigned long long* slot, int s) { slot[s] = kEmpty; }
};

template <>
struct Table<false> {
  static constexpr int kTile = kTileF64;
  static constexpr int kHalf = kSlots / 2;   // keys below, FP64 sums above
  static __device__ __forceinline__ void insert(unsigned long long* slot, int32_t* ncl, uint16_t* claimed, int j,
                                                int32_t c, double w) {
    const unsigned long long key = ((unsigned long long)j << 32) | (uint32_t)c;
    double* sum = reinterpret_cast<double*>(slot + kHalf);
    uint32_t h = (uint32_t)((key * 0x9E3779B97F4A7C15ull) >> (64 - 12));
    for (int p = 0; p < kHalf; ++p) {
      const unsigned long long prev = atomicCAS(&slot[h], kEmpty, key);
      if (prev == kEmpty) claimed[atomicAdd(ncl, 1)] = (uint16_t)h;
      if (prev == kEmpty || prev == key) { atomicAdd(&sum[h], w); return; }
      h = (h + 1) & (kHalf - 1);
    }
  }
  static __device__ __forceinline__ void get(const unsigned long long* slot, int s, int& j, int32_t& c, double& w) {
    const unsigned long long key = slot[s];
    j = (int)(key >> 32);
    c = (int32_t)(uint32_t)key;
    w = reinterpret_cast<const double*>(slot + kHalf)[s];
  }
  static __device__ __forceinline__ void clear(unsigned long long* slot, int s) {
    slot[s] = kEmpty;
    reinterpret_cast<double*>(slot + kHalf)[s] = 0.0;
  }
};

// A later pass: rows hashed tile by tile.
template <int NT, bool INT>
__device__ void moves_hash(const Team<NT>& T, Smem<NT>& S, const Work& W, const List& L, int32_t v, int32_t vend) {
  using Tab = Table<INT>;
  constexpr int kItems = Tab::kTile / NT;
  constexpr int kTabSlots = INT ? kSlots : kSlots / 2;
  unsigned long long* slot = S.u.slot;
  for (int s = T.tid; s < kTabSlots; s += NT) Tab::clear(slot, s);
  if (T.tid == 0) S.nclaimed = 0;
  __syncthreads();
  while (v < vend) {
    const int nv = tile_rows<NT>(W.roff, v, vend, Tab::kTile);
    if (nv == 0) return;   // cannot happen, as above
    const int32_t base = W.roff[v];
    const int n = W.roff[v + nv] - base;
    if (n > 0) {
      for (int j = T.tid; j < nv; j += NT) {
        S.own[j] = W.comm[v + j];
        S.kf[j] = W.kfrac[v + j];
        S.bestg[j] = 0ull;
        S.bestc[j] = kNone;
        S.nseg[j] = 0;
      }
      int jj[kItems];
      int32_t cc[kItems];
      double wd[kItems];
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        const int x = q * NT + T.tid;
        jj[q] = -1;
        cc[q] = 0;
        wd[q] = 0.0;
        if (x < n) {
          const int32_t u = L.src[base + x], d = L.dst[base + x];
          if (u != d) jj[q] = u - v;
          cc[q] = d;
          wd[q] = merged_w(L.w[base + x]);
        }
      }
#pragma unroll
      for (int q = 0; q < kItems; ++q)
        if (jj[q] >= 0) cc[q] = W.comm[cc[q]];
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        if (jj[q] >= 0) {
          if (cc[q] == S.own[jj[q]]) atomicOr(&S.nseg[jj[q]], 1 << 30);
          Tab::insert(slot, &S.nclaimed, S.claimed, jj[q], cc[q], wd[q]);
        }
      }
      __syncthreads();
      const int nc = S.nclaimed;
      double gg[kItems];
#pragma unroll
      for (int q = 0; q < kItems; ++q) {       // count, best gain bits
        const int x = q * NT + T.tid;
        gg[q] = 0.0;
        jj[q] = -1;
        if (x < nc) {
          Tab::get(slot, S.claimed[x], jj[q], cc[q], wd[q]);
          atomicAdd(&S.nseg[jj[q]], 1);
          if (wd[q] != 0.0) gg[q] = __dsub_rn(wd[q], __dmul_rn(W.tot[cc[q]], S.kf[jj[q]]));
          if (gg[q] > 0.0) atomicMax(&S.bestg[jj[q]], (unsigned long long)__double_as_longlong(gg[q]));
          Tab::clear(slot, S.claimed[x]);
        }
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q)         // smallest community among the best gains
        if (jj[q] >= 0 && gg[q] > 0.0 && (unsigned long long)__double_as_longlong(gg[q]) == S.bestg[jj[q]])
          atomicMin(&S.bestc[jj[q]], cc[q]);
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q)
        if (jj[q] >= 0 && cc[q] == S.bestc[jj[q]]) S.bestw[jj[q]] = wd[q];
      if (T.tid == 0) S.nclaimed = 0;
      __syncthreads();
      for (int j = T.tid; j < nv; j += NT) {
        const int32_t i = v + j;
        if (W.roff[i + 1] > W.roff[i]) {
          const int32_t c = S.bestc[j], s = S.nseg[j];
          const int32_t nseg = (s & ((1 << 30) - 1)) + ((W.hasl[i] && !(s >> 30)) ? 1 : 0);
          decide<false>(W, i, S.own[j], c, c == kNone ? 0.0 : S.bestw[j], nseg);
        }
      }
      __syncthreads();
    }
    v += nv;
  }
}

// Commit of a pass (communitySetKernel) with the Q partials of the new state.
template <int NT>
__device__ __forceinline__ void commit(const Team<NT>& T, Smem<NT>& S, const Work& W, int32_t V, double m) {
  const double twom = __dmul_rn(2.0, m);
  group_partials<NT>(T, S, V, W.qpart, [&](int64_t c) {
    double t = W.tot[c], x = W.in[c];
    int32_t sz = W.size[c];
    delta_commit(W.delta[c], W.k[c], t, x, sz);
    W.tot[c] = t;
    W.in[c] = x;
    W.size[c] = sz;
    W.comm[c] = W.next[c];
    return q_term(x, t, m, twom);
  });
}

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Entries of the list checked: ids and weights, strict order, and symmetry by
// the fingerprints of list_check_kernel.
template <int NT>
__device__ void check_list(const Team<NT>& T, const Work& W, const List& L, int64_t E, int32_t V) {
  const uint64_t K1 = 0x243F6A8885A308D3ull, K2 = 0x13198A2E03707344ull;
  const unsigned full = 0xffffffffu;
  uint64_t d1 = 0, d2 = 0;
  uint32_t f = 0;
  for (int64_t e = T.gt(); e < E; e += T.stride()) {
    const int32_t u = L.src[e], v = L.dst[e];
    const float x = L.w[e];
    if (!entry_ok(u, v, x, V)) f |= fBad;
    if (e > 0) {
      const int32_t u0 = L.src[e - 1], v0 = L.dst[e - 1];
      if (!(u > u0 || (u == u0 && v > v0))) f |= fUnsorted;
    }
    if (u != v) {
      const uint32_t wb = __float_as_uint(x);
      d1 += edge_hash((uint32_t)u, (uint32_t)v, wb, K1) - edge_hash((uint32_t)v, (uint32_t)u, wb, K1);
      d2 += edge_hash((uint32_t)u, (uint32_t)v, wb, K2) - edge_hash((uint32_t)v, (uint32_t)u, wb, K2);
    }
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    d1 += __shfl_down_sync(full, d1, o);
    d2 += __shfl_down_sync(full, d2, o);
  }
  f = __reduce_or_sync(full, f);
  if ((T.tid & 31) == 0) {
    if (d1) atomicAdd(&W.ctl->sums[0], (unsigned long long)d1);
    if (d2) atomicAdd(&W.ctl->sums[1], (unsigned long long)d2);
    if (f) atomicOr(&W.ctl->check, f);
  }
}

// The coarse list of the level under W.part (C communities) into (osrc, odst,
// ow); returns its length.  Stable LSD sort of the entries' keys over the
// cluster: block r owns the r-th share of the positions, counts its digits,
// and places its keys after those of all blocks before it.
template <int NT>
__device__ int64_t coarsen(const Team<NT>& T, Smem<NT>& S, const Work& W, const List& L, int64_t E, int32_t C,
                           int32_t* osrc, int32_t* odst, float* ow) {
  constexpr int kIt = 4;
  const unsigned full = 0xffffffffu;
  const int lane = T.tid & 31, wid = T.tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  int b = 1;
  while (b < kCommBits && (1 << b) < C) ++b;
  const int bits = 2 * b, np = (bits + 7) / 8, width = (bits + np - 1) / np;
  const uint32_t dmask = (1u << width) - 1u;
  const int64_t s0 = E * T.rank / T.K, s1 = E * (T.rank + 1) / T.K;
  int cur = 0;
  for (int p = 0; p < np; ++p) {
    for (int x = T.tid; x < kDigits; x += NT) S.hist[x] = 0;
    __syncthreads();
    for (int64_t e = s0 + T.tid; e < s1; e += NT) {
      uint32_t key;
      if (p == 0) {
        key = ((uint32_t)W.part[L.src[e]] << b) | (uint32_t)W.part[L.dst[e]];
        const float x = L.w[e];
        W.key[0][e] = key;
        W.val[0][e] = x == 0.0f ? 1.0f : x;       // InducedGraphKernel.cu:38-39
        W.wsum[e] = 0.0;
      } else {
        key = W.key[cur][e];
      }
      atomicAdd(&S.hist[(key >> (p * width)) & dmask], 1u);
    }
    __syncthreads();
    for (int x = T.tid; x < kDigits; x += NT) W.ghist[x * T.K + T.rank] = S.hist[x];
    T.sync();
    uint32_t tot = 0, pre = 0;
    if (T.tid < kDigits)
      for (int r = 0; r < T.K; ++r) {
        const uint32_t c = W.ghist[T.tid * T.K + r];
        if (r < T.rank) pre += c;
        tot += c;
      }
    uint32_t all;
    const uint32_t ex = block_excl<NT>(tot, S.wtot, &all);
    if (T.tid < kDigits) S.dbase[T.tid] = ex + pre;
    for (int64_t t0 = s0; t0 < s1; t0 += NT * kIt) {
      for (int x = T.tid; x < (NT / 32) * (kDigits + 1); x += NT) (&S.u.wc[0][0])[x] = 0;
      __syncthreads();
      uint32_t key[kIt], rank[kIt], dg[kIt];
      float val[kIt];
      const int64_t base = t0 + (int64_t)wid * 32 * kIt;
#pragma unroll
      for (int j = 0; j < kIt; ++j) {
        const int64_t i = base + j * 32 + lane;
        key[j] = i < s1 ? W.key[cur][i] : 0u;
        val[j] = i < s1 ? W.val[cur][i] : 0.0f;
        dg[j] = i < s1 ? (key[j] >> (p * width)) & dmask : (uint32_t)kDigits;
      }
#pragma unroll
      for (int j = 0; j < kIt; ++j) {
        const unsigned peers = __match_any_sync(full, dg[j]);
        const uint32_t before = S.u.wc[wid][dg[j]];
        rank[j] = before + __popc(peers & lt);
        __syncwarp();
        if ((peers & lt) == 0) S.u.wc[wid][dg[j]] = before + __popc(peers);
        __syncwarp();
      }
      __syncthreads();
      if (T.tid < kDigits) {
        uint32_t run = S.dbase[T.tid];
        for (int w = 0; w < NT / 32; ++w) {
          const uint32_t c = S.u.wc[w][T.tid];
          S.u.wc[w][T.tid] = run;
          run += c;
        }
        S.dbase[T.tid] = run;
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < kIt; ++j)
        if (dg[j] < (uint32_t)kDigits) {
          const uint32_t o = S.u.wc[wid][dg[j]] + rank[j];
          W.key[cur ^ 1][o] = key[j];
          W.val[cur ^ 1][o] = val[j];
        }
      __syncthreads();
    }
    T.sync();
    cur ^= 1;
  }
  // runs of equal keys: heads counted per block, then each run's pieces added
  const uint32_t* key = W.key[cur];
  const float* val = W.val[cur];
  uint32_t heads = 0;
  for (int64_t i0 = s0; i0 < s1; i0 += NT) {
    const int64_t i = i0 + T.tid;
    heads += __syncthreads_count(i < s1 && (i == 0 || key[i] != key[i - 1]));
  }
  if (T.tid == 0) W.ctl->count[1][T.rank] = heads;
  T.sync();
  uint32_t run = 0, cnt = 0;
  for (int r = 0; r < T.K; ++r) {
    const uint32_t c = W.ctl->count[1][r];
    if (r < T.rank) run += c;
    cnt += c;
  }
  const uint32_t cmask = (1u << b) - 1u;
  for (int64_t t0 = s0; t0 < s1; t0 += NT * kIt) {
    const int64_t i0 = t0 + (int64_t)T.tid * kIt;
    uint32_t k[kIt + 1], hm = 0;
    k[0] = i0 > 0 && i0 < s1 ? key[i0 - 1] : 0u;
#pragma unroll
    for (int j = 0; j < kIt; ++j) {
      k[j + 1] = i0 + j < s1 ? key[i0 + j] : 0u;
      if (i0 + j < s1 && (i0 + j == 0 || k[j + 1] != k[j])) hm |= 1u << j;
    }
    uint32_t all;
    uint32_t r = run + block_excl<NT>((uint32_t)__popc(hm), S.wtot, &all);   // runs started before the thread
    run += all;
    double s = 0.0;
    bool any = false;
#pragma unroll
    for (int j = 0; j < kIt; ++j) {
      if (i0 + j < s1) {
        if ((hm >> j) & 1u) {
          if (any) atomicAdd(&W.wsum[r - 1], s);
          s = 0.0;
          osrc[r] = (int32_t)(k[j + 1] >> b);
          odst[r] = (int32_t)(k[j + 1] & cmask);
          ++r;
        }
        s = __dadd_rn(s, (double)val[i0 + j]);
        any = true;
      }
    }
    if (any) atomicAdd(&W.wsum[r - 1], s);
  }
  T.sync();
  for (int64_t i = T.gt(); i < cnt; i += T.stride()) ow[i] = __double2float_rn(W.wsum[i]);
  return (int64_t)cnt;
}

template <int NT>
__global__ void __launch_bounds__(NT) small_kernel(const SmallJob* jobs, int K, SmallCfg cfg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem<NT>& S = *reinterpret_cast<Smem<NT>*>(smem_raw);
  const SmallJob J = jobs[blockIdx.x / K];
  const Team<NT> T{K, (int)(blockIdx.x % K), (int)threadIdx.x};
  Work W;
  carve(J.work, J.V, J.E, W);
  const bool lead = T.rank == 0 && T.tid == 0;
  List L{J.src, J.dst, J.w};
  int32_t V = J.V;
  int64_t E = J.E;
  int32_t ncomms = 0;
  int buf = -1, nlev = 0, status = LVG_OK;
  bool open = false, symmetric = J.check == 0, bad = false;
  double mod = J.mod, lower = 0.0;
  int64_t part_off = 0;
  for (;;) {
    unsigned long long t0 = lead ? now_ns() : 0ull;
    const int level = J.level0 + nlev;
    if (nlev >= kSmallLevels || (J.parts && part_off + 2 * (int64_t)V > J.parts_cap)) { open = true; break; }
    // ---- build
    for (int32_t i = T.gt(); i < V; i += T.stride()) {
      W.k[i] = 0.0;
      W.loopw[i] = 0.0f;
      W.hasl[i] = 0;
    }
    if (lead) {
      W.ctl->flags = W.ctl->flags2 = W.ctl->check = W.ctl->loops = 0u;
      W.ctl->sums[0] = W.ctl->sums[1] = 0ull;
    }
    T.sync();
    if (!symmetric) {
      check_list<NT>(T, W, L, E, V);
      T.sync();
      const uint32_t f = W.ctl->check;
      if (f & fBad) { bad = true; break; }
      if (f != 0u || W.ctl->sums[0] != 0ull || W.ctl->sums[1] != 0ull) { open = true; break; }
    }
    {
      uint32_t f = 0, nl = 0;
      for (int64_t e0 = (int64_t)T.rank * NT; e0 < E; e0 += T.stride()) {
        const int64_t e = e0 + T.tid;
        const bool in = e < E;
        const int32_t u = in ? L.src[e] : -1, d = in ? L.dst[e] : -2;
        const float x = in ? L.w[e] : 0.0f;
        if (in) {
          const int32_t up = e > 0 ? L.src[e - 1] : -1;
          for (int32_t r = up + 1; r <= u; ++r) W.roff[r] = (int32_t)e;
          if (e == E - 1)
            for (int32_t r = u + 1; r <= V; ++r) W.roff[r] = (int32_t)E;
          if (x != truncf(x)) f |= fNotInt;
          if (u == d) { W.loopw[u] = x; W.hasl[u] = 1; ++nl; }
        }
        float g = x == 0.0f ? 1.0f : x;             // InitKernel.cu:165-170, both copies of the entry
        if (u == d) g *= 2.0f;
        const double s = seg_warp_sum<int32_t>(in ? __dadd_rn((double)g, (double)g) : 0.0, u);
        if (seg_warp_last<int32_t>(u, in)) atomicAdd(&W.k[u], s);
      }
      f = __reduce_or_sync(0xffffffffu, f);
      nl = __reduce_add_sync(0xffffffffu, nl);
      if ((T.tid & 31) == 0) {
        if (f) atomicOr(&W.ctl->flags, f);
        if (nl) atomicAdd(&W.ctl->loops, nl);
      }
      group_partials<NT>(T, S, E, W.mpart, [&](int64_t e) { return (double)L.w[e]; });   // NeighbourCompute.cu:46
    }
    T.sync();
    const bool integral = !(W.ctl->flags & fNotInt);
    symmetric = integral;   // of the next list: exact sums round alike in both directions
    const int64_t nnz = E - (int64_t)W.ctl->loops;
    const double m = finish_sum<NT>(S, W.mpart, E);
    const double twom = __dmul_rn(2.0, m);
    {
      const int32_t longest = integral ? kTileInt : kTileF64;
      uint32_t f = 0;
      group_partials<NT>(T, S, V, W.qpart, [&](int64_t i) {
        const double k = W.k[i], x = (double)W.loopw[i];
        W.comm[i] = (int32_t)i;                 // InitKernel.cu:213-215
        W.next[i] = (int32_t)i;
        W.tot[i] = k;                           // InitKernel.cu:236
        W.in[i] = x;                            // InitKernel.cu:242
        W.size[i] = 1;                          // OneLevelKernel.cu:87
        delta_clear(W.delta[i]);
        W.cand[i] = -1;
        W.kfrac[i] = m > 0.0 ? __ddiv_rn(k, twom) : 0.0;   // OneLevelKernel.cu:307
        W.minidx[i] = kNone;
        if (W.roff[i + 1] - W.roff[i] > longest) f |= fUnfit;
        if (!(k < 1073741824.0)) f |= fNotInt;
        return q_term(x, k, m, twom);
      });
      if (f) atomicOr(&W.ctl->flags2, f);
    }
    T.sync();
    const uint32_t f2 = W.ctl->flags2;
    const bool packed = integral && !(f2 & fNotInt);
    // sums beyond 32 bits take the FP64 tiles, whose rows are shorter
    if ((f2 & fUnfit) || (integral && !packed)) { open = true; break; }
    const double q0 = finish_sum<NT>(S, W.qpart, V);
    lower = level == 0 ? q0 : mod;              // LouvainCPP.cpp:356,446
    const int32_t v0 = row_at(W.roff, V, E * T.rank / T.K);
    const int32_t v1 = T.rank == T.K - 1 ? V : row_at(W.roff, V, E * (T.rank + 1) / T.K);
    unsigned long long t1 = lead ? now_ns() : 0ull;
    // ---- passes
    double q_prev = q0, floor_q = -1.0;         // curMod = -1 (OneLevelKernel.cu:528)
    int pass = 1, st = LVG_OK;
    float pass_ms[2] = {0.0f, 0.0f};
    for (;; ++pass) {
      const unsigned long long p0 = lead ? now_ns() : 0ull;
      if (pass == 1) moves_first<NT>(T, S, W, L, v0, v1);
      else if (packed) moves_hash<NT, true>(T, S, W, L, v0, v1);
      else moves_hash<NT, false>(T, S, W, L, v0, v1);
      T.sync();
      if (lead && pass <= 2) pass_ms[pass - 1] = (float)(now_ns() - p0) * 1e-6f;
      const bool stop = __dsub_rn(q_prev, floor_q) < cfg.pass_min;             // OneLevelKernel.cu:889-896
      const bool capped = cfg.max_passes >= 0 && pass >= cfg.max_passes;
      if (stop || capped) {
        for (int32_t i = T.gt(); i < V; i += T.stride()) delta_clear(W.delta[i]);
        st = stop ? LVG_OK : LVG_ERR_NOT_CONVERGED;
        break;
      }
      commit<NT>(T, S, W, V, m);
      T.sync();
      const double q = finish_sum<NT>(S, W.qpart, V);
      floor_q = q_prev < lower ? lower : q_prev;
      q_prev = q;
      if (pass >= kSmallPassCap) { open = true; break; }
    }
    if (open) break;
    T.sync();
    for (int32_t i = T.gt(); i < V; i += T.stride()) {      // isolated merge (OneLevelKernel.cu:138-171)
      const int32_t c = W.cand[i];
      if (c >= 0) {
        W.next[i] = c;
        move_deltas<false>(W.delta, W.comm[i], c, W.k[i], __dadd_rn(0.0, (double)W.loopw[i]));
      }
    }
    T.sync();
    commit<NT>(T, S, W, V, m);
    T.sync();
    const double ql = finish_sum<NT>(S, W.qpart, V);
    unsigned long long t2 = lead ? now_ns() : 0ull;
    // ---- renumber by smallest member (RenumberKernel.cu:121-133)
    for (int32_t i = T.gt(); i < V; i += T.stride()) atomicMin(&W.minidx[W.comm[i]], i);
    T.sync();
    const int32_t i0 = (int32_t)((int64_t)V * T.rank / T.K), i1 = (int32_t)((int64_t)V * (T.rank + 1) / T.K);
    uint32_t heads = 0;
    for (int32_t b0 = i0; b0 < i1; b0 += NT) {
      const int32_t i = b0 + T.tid;
      heads += __syncthreads_count(i < i1 && W.minidx[W.comm[i < i1 ? i : i0]] == i);
    }
    if (T.tid == 0) W.ctl->count[0][T.rank] = heads;
    T.sync();
    uint32_t run = 0, C = 0;
    for (int r = 0; r < T.K; ++r) {
      const uint32_t c = W.ctl->count[0][r];
      if (r < T.rank) run += c;
      C += c;
    }
    for (int32_t b0 = i0; b0 < i1; b0 += NT) {
      const int32_t i = b0 + T.tid;
      const int32_t c = i < i1 ? W.comm[i] : 0;
      const bool h = i < i1 && W.minidx[c] == i;
      uint32_t all;
      const uint32_t ex = block_excl<NT>(h ? 1u : 0u, S.wtot, &all);
      if (h) W.newid[c] = (int32_t)(run + ex);
      run += all;
    }
    T.sync();
    for (int32_t i = T.gt(); i < V; i += T.stride()) {
      const int32_t c = W.comm[i], id = W.newid[c];
      W.part[i] = id;
      if (J.parts) {
        J.parts[part_off + i] = id;
        J.parts[part_off + V + i] = c;
      }
    }
    for (int32_t i = T.gt(); i < J.V; i += T.stride())       // partitionAtLevel (LouvainCPP.cpp:82-106)
      J.comp[i] = W.newid[W.comm[nlev == 0 ? i : J.comp[i]]];
    T.sync();
    unsigned long long t3 = lead ? now_ns() : 0ull;
    // ---- level break (LouvainCPP.cpp:466)
    bool last = false;
    if (st != LVG_OK) { status = st; last = true; }
    else if (level > 0 && (ql - mod) < cfg.level_min) last = true;
    else if (cfg.max_levels >= 0 && level + 1 >= cfg.max_levels) { status = LVG_ERR_NOT_CONVERGED; last = true; }
    mod = ql;
    int64_t E1 = 0;
    int32_t *ns = nullptr, *nd = nullptr;
    float* nw = nullptr;
    if (!last) {
      list_of(J.lists, J.E, nlev & 1, &ns, &nd, &nw);
      E1 = coarsen<NT>(T, S, W, L, E, (int32_t)C, ns, nd, nw);
    }
    if (lead && J.lv) {
      SmallLevel& R = J.lv[nlev];
      R.V = V;
      R.C = (int32_t)C;
      R.passes = pass;
      R.E = E;
      R.nnz = nnz;
      R.q_start = q0;
      R.q_level = ql;
      R.ms[0] = (float)(t1 - t0) * 1e-6f;
      R.ms[1] = (float)(t2 - t1) * 1e-6f;
      R.ms[2] = (float)(t3 - t2) * 1e-6f;
      R.ms[3] = last ? 0.0f : (float)(now_ns() - t3) * 1e-6f;
      R.pass_ms[0] = pass_ms[0];
      R.pass_ms[1] = pass_ms[1];
      R.part_off = part_off;
    }
    part_off += 2 * (int64_t)V;
    ncomms = (int32_t)C;
    ++nlev;
    if (last) break;
    buf = (nlev - 1) & 1;
    L = List{ns, nd, nw};
    V = (int32_t)C;
    E = E1;
  }
  double q_final = 0.0;
  if (J.want_q && !open && !bad) {
    // Newman modularity of comp over the job's list, as nm_accum_sym_kernel:
    // the list is symmetric, so each entry adds 2w to its source's community
    const int64_t C = ncomms;
    for (int64_t i = T.gt(); i < C; i += T.stride()) W.tot[i] = W.in[i] = 0.0;
    T.sync();
    for (int64_t e0 = (int64_t)T.rank * NT; e0 < J.E; e0 += T.stride()) {
      const int64_t e = e0 + T.tid;
      const bool in = e < J.E;
      const int32_t u = in ? J.src[e] : -1;
      const double x = in ? 2.0 * (double)J.w[e] : 0.0;
      const int32_t a = in ? J.comp[u] : -1, b = in ? J.comp[J.dst[e]] : -1;
      const double kin = seg_warp_sum<int32_t>(x, u);
      const double ain = seg_warp_sum<int32_t>(a == b ? x : 0.0, u);
      if (seg_warp_last<int32_t>(u, in)) {
        atomicAdd(&W.tot[a], kin);
        if (ain != 0.0) atomicAdd(&W.in[a], ain);
      }
    }
    T.sync();
    group_partials<NT>(T, S, C, W.mpart, [&](int64_t c) { return W.tot[c]; });
    T.sync();
    const double tw = finish_sum<NT>(S, W.mpart, C);
    group_partials<NT>(T, S, C, W.qpart, [&](int64_t c) {
      const double f = __ddiv_rn(W.tot[c], tw);
      return tw > 0.0 ? __dsub_rn(__ddiv_rn(W.in[c], tw), __dmul_rn(f, f)) : 0.0;
    });
    T.sync();
    q_final = finish_sum<NT>(S, W.qpart, C);
  }
  if (lead) {
    SmallResult& O = *J.res;
    O.n_levels = nlev;
    O.n_comms = ncomms;
    O.open = open ? 1 : 0;
    O.status = status;
    O.bad = bad ? 1 : 0;
    O.V = V;
    O.buf = buf;
    O.E = E;
    O.mod = mod;
    O.lower = lower;
    O.q_final = q_final;
  }
}

template <int NT>
void set_attributes() {
  constexpr int kDevs = 64;
  static std::mutex mu;
  static bool done[kDevs] = {};
  int dev = 0;
  LVG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (dev >= 0 && dev < kDevs && done[dev]) return;
  LVG_CUDA(cudaFuncSetAttribute(small_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem<NT>)));
  LVG_CUDA(cudaFuncSetAttribute(small_kernel<NT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  if (dev >= 0 && dev < kDevs) done[dev] = true;
}

template <int NT>
void launch(const SmallJob* jobs, int n, int K, const SmallCfg& cfg, cudaStream_t s) {
  set_attributes<NT>();
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)(n * K));
  lc.blockDim = dim3(NT);
  lc.dynamicSmemBytes = sizeof(Smem<NT>);
  lc.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)K;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  lc.attrs = at;
  lc.numAttrs = K > 1 ? 1 : 0;
  LVG_CUDA(cudaLaunchKernelEx(&lc, small_kernel<NT>, jobs, K, cfg));
  count_launch();
}

}  // namespace

size_t small_list_bytes(int64_t E) { return 6 * up256(4 * (size_t)E); }

size_t small_work_bytes(int32_t V, int64_t E) {
  Work W;
  return carve(nullptr, V, E, W);
}

void small_list(char* lists, int64_t E, int buf, int32_t** src, int32_t** dst, float** w) {
  list_of(lists, E, buf, src, dst, w);
}

bool small_fits(int64_t V, int64_t E, int64_t max_entries) {
  return V > 0 && V <= kSmallMaxV && E > 0 && E <= max_entries;
}

void small_run(const SmallJob* d_jobs, int n, int K, const SmallCfg& cfg, cudaStream_t s) {
  if (n <= 0) return;
  if (K >= 8) launch<1024>(d_jobs, n, K, cfg, s);
  else launch<512>(d_jobs, n, K, cfg, s);
}

}  // namespace lvg
