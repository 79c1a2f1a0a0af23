// Small graphs: all levels of a dendrogram inside a few launches.
//
// The level kernels take about 70 launches and 17 host reads of sizes a
// level, some 0.7 ms however small the level is.  Here the level loop runs
// inside a kernel: the phases of a level are separated by barriers instead of
// launches, every decision of the loop (the ΔQ test, the level break, sizes) is
// taken by all threads from the same values, and the host reads one result at
// the end.  The launches of a run, queued one behind the other:
//   small_kernel       a cooperative grid, a block an SM, while a level has
//                      more than 64 Ki entries and vertices (a single run's;
//                      its barrier counts arrivals in device memory)
//   small_kernel       a thread-block cluster (hardware barriers) below that;
//                      in a batch each graph has its own, of one block to
//                      eight, so that its levels need not wait for the others
//   small_tail_kernel  one block, once a level fits its shared memory
//   small_sum_kernel, small_end_kernel   the final modularity and the result
//
// Where a level's list is strictly sorted by (src, dst) and symmetric, a row is
// a contiguous range of the list and the merged CSR entry of (u, v, w) is
// (u, v, 2w); no CSR is written.  Other lists (coarse ones of a graph whose
// edges are listed once) have the doubled list sorted and merged into a CSR
// first.  The rules are the level kernels' (rules.cuh):
//   build    row starts, degrees and self loops from one pass over the list,
//            m and every Q on the fixed tree
//   pass 1   singletons: the best candidate of a row is an argmax over its
//            entries (segmented warp argmax, then shared-memory max / min)
//   pass 2+  tiles of consecutive rows hashed as (row, community) pairs in
//            shared memory: 32-bit keys and sums when the weights are whole and
//            no degree reaches 2^30, key + FP64 sum otherwise; rows longer than a tile in tables in
//            device memory, by all blocks
//   renumber by smallest member; coarse keys (cu << b | cv) sorted by a stable
//            LSD radix sort across the blocks, runs summed in FP64 (by one
//            block and few communities: a sum for every pair of them)
// A list in any order without room for its CSR, or more levels or passes than
// the tables hold, end the launch with the level left open; the caller goes on
// with the level kernels from the same list.
#include <algorithm>
#include <atomic>
#include <cooperative_groups.h>
#include <mutex>
#include <type_traits>

#include "prims.cuh"
#include "rules.cuh"
#include "small.cuh"

namespace lvg {
namespace {

namespace cg = cooperative_groups;

constexpr int kItems = 4;                  // entries of a tile per thread
// Tile of a block of NT threads: entries, slots (16 or 8 bytes an entry, at
// most half full), and rows (10 bits of a packed key).
template <int NT>
struct Tile {
  static constexpr int kInt = kItems * NT;       // entries, packed slots
  static constexpr int kSlots = 2 * kInt;
  static constexpr int kF64 = kInt / 2;          // entries, key and sum in two slots
  static constexpr int kRows = NT;
  static constexpr int kLog = NT == 1024 ? 13 : 12;
  static_assert(kSlots == 1 << kLog && kRows <= 1 << 10, "tile sizes");
};
constexpr int kCommBits = 18;              // community bits of a packed key
constexpr int kDigits = 256;
constexpr int64_t kGridEntries = 4096;     // grid mode: entries a block, at least
constexpr int kShortRow = kItems * 512 / 2;   // the smaller blocks' FP64 tile: no row up to this is long
constexpr int kGaps = 64;                  // runs of empty rows a block fills together
constexpr int kHubs = 32;                  // long rows a block looks up at a time
constexpr int kResThreads = 512;
constexpr int kResV = 512, kResE = 6144;   // a level this small lives in one block's shared memory
constexpr unsigned long long kEmpty = ~0ull;
static_assert(kSmallMaxV <= (1 << kCommBits), "packed keys hold 18-bit communities");

enum : uint32_t { fNotInt = 1u, fBad = 4u, fUnsorted = 8u, fLong = 16u };
// kPhaseMid: the grid left the level to a cluster; kPhaseTail: a level fits
// one block's shared memory; kPhaseEnd: the levels are done.
enum : int32_t { kPhaseNone = 0, kPhaseMid = 1, kPhaseTail = 2, kPhaseEnd = 3 };
enum : int32_t { kCompDone = 0, kCompTail = 1, kCompTailAll = 2 };

// Control words of a level's blocks.
struct Ctl {
  uint32_t flags, flags2, check, loops;
  uint32_t nlong;               // rows in Work::longs
  unsigned long long sums[2];
  uint32_t count[2][kSmallMaxBlocks];
  unsigned long long arrived;   // grid barrier: arrivals so far
  uint32_t dead;                // grid barrier: a wait ran out
};

// Where the levels of a job stand between its launches.
struct Between {
  int32_t phase;             // kPhase*
  int32_t nlev, buf, symmetric;
  int32_t V, ncomms, open, bad, status;
  int32_t comp;              // kComp*: what the composition still needs
  int64_t E, part_off;
  double mod;
  double ms_per_tick;
};

struct Work {
  Ctl* ctl;
  Between* bt;
  double *k, *kfrac, *tot, *in, *qpart, *mpart;
  Delta* delta;
  int32_t *roff, *comm, *next, *cand, *size, *minidx, *newid;
  float* loopw;
  int32_t* hasl;
  uint64_t* key[2];
  uint32_t* ghist;
  int32_t* rc;               // composition of the resident levels
  float* val[2];
  double* wsum;
  int32_t* longs;            // rows longer than a tile of FP64 sums
  int32_t *csrc, *cdst;      // CSR of a list that is not symmetric, row by row
  float* cw;
};

__host__ __device__ inline size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

// dbl: room for the doubled list of a level and the CSR made from it.
// blocks: of the job's team, at most (one has no counts to share).
__host__ __device__ inline size_t carve(char* base, int64_t V, int64_t E, bool dbl, int blocks, Work& W) {
  size_t o = 0;
  const int64_t n = dbl ? 2 * E : E;
  auto take = [&](size_t bytes) {
    char* p = base + o;
    o += up256(bytes);
    return p;
  };
  W.ctl = (Ctl*)take(sizeof(Ctl));
  W.bt = (Between*)take(sizeof(Between));
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
  W.loopw = (float*)take(4 * V);
  W.hasl = (int32_t*)take(4 * V);
  W.key[0] = (uint64_t*)take(8 * n);
  W.key[1] = (uint64_t*)take(16 * n);   // wsum behind it: together the sums of the long rows' tables
  W.wsum = (double*)W.key[1] + n;
  W.val[0] = (float*)take(4 * n);
  W.val[1] = (float*)take(4 * n);
  W.csrc = dbl ? (int32_t*)take(4 * n) : nullptr;
  W.cdst = dbl ? (int32_t*)take(4 * n) : nullptr;
  W.cw = dbl ? (float*)take(4 * n) : nullptr;
  W.longs = (int32_t*)take(4 * (n / kShortRow + 1));
  W.ghist = (uint32_t*)take(blocks > 1 ? 4 * kDigits * blocks : 0);
  W.rc = (int32_t*)take(4 * kResV);
  return o;
}

__host__ __device__ inline void list_of(char* lists, int64_t E, int buf, int32_t** src, int32_t** dst, float** w) {
  char* p = lists + (size_t)buf * 3 * up256(4 * E);
  *src = (int32_t*)p;
  *dst = (int32_t*)(p + up256(4 * E));
  *w = (float*)(p + 2 * up256(4 * E));
}

// A resident level: its list and per-vertex arrays in shared memory, under
// the names Work gives their device-memory counterparts.
struct Resident {
  int32_t src[kResE], dst[kResE];
  float w[kResE];
  Delta delta[kResV];
  double k[kResV], kfrac[kResV], tot[kResV], in[kResV], qpart[1], mpart[kResE / kGroup + 1];
  int32_t roff[kResV + 1], comm[kResV], next[kResV], cand[kResV], size[kResV], minidx[kResV], newid[kResV],
      hasl[kResV], comp[kResV];
  float loopw[kResV];
  Ctl ctl[1];
  uint64_t* key[2];          // device memory (levels of more communities than `cell` holds pairs for)
  uint32_t* ghist;
  float* val[2];
  double* wsum;
};
static_assert(kResV < kGroup, "one group of communities");

// Working space of a block of NT threads.
template <int NT, int CELLS>
struct Space {
  static constexpr int kSlots = Tile<NT>::kSlots, kTileRows = Tile<NT>::kRows, kTileInt = Tile<NT>::kInt;
  union {
    unsigned long long slot[kSlots];
    struct {
      uint32_t wc[NT / 32][kDigits];     // a warp's keys of each digit
      uint32_t meet[NT / 32][kDigits];   // its lanes that hold one
    } sort;
    uint32_t part[2][NT / kDigits][kDigits];
    double stage[kGroup];
    double cell[CELLS];        // sums of a coarse graph of few communities
  } u;
  uint32_t besth[kTileRows], bestl[kTileRows];   // best gain, upper and lower half
  double bestw[kTileRows];
  double kf[kTileRows];
  int32_t bestc[kTileRows];
  int32_t own[kTileRows];
  int32_t nseg[kTileRows];   // distinct candidate communities; bit 30: own community seen
  uint16_t claimed[kTileInt];
  uint32_t hist[kDigits];
  uint32_t dbase[kDigits];
  double ws[8];
  double bcast;
  uint32_t wtot[NT / 32];
  double rg[NT / 32], rw[NT / 32];   // long rows: each warp's best candidate
  int32_t rc[NT / 32];
  int32_t nhub, hub[kHubs];
  int32_t ngap;
  int4 gap[kGaps];
  int32_t nclaimed, row0, row1;
  unsigned long long goal;   // grid barrier: arrivals awaited
  unsigned long long wait_ns;   // and the limit of the wait
  int32_t alive;
  SmallJob J;
};

extern __shared__ __align__(16) unsigned char smem_raw[];

// A job's levels by several blocks, or one, over device memory.
template <int NT_>
struct Multi {
  static constexpr int NT = NT_;
  static constexpr bool kResident = false;
  static constexpr int kCells = 1;
  struct Smem {
    Space<NT, kCells> s;
    Work w;                  // read from here, not held in registers
  };
  static __device__ __forceinline__ Smem& mem() { return *reinterpret_cast<Smem*>(smem_raw); }
  static __device__ __forceinline__ Space<NT, kCells>& S() { return mem().s; }
  static __device__ __forceinline__ Work& W() { return mem().w; }
};

// The last levels of a job by one block over its shared memory.
struct Tail {
  static constexpr int NT = kResThreads;
  static constexpr bool kResident = true;
  static constexpr int kCells = 8192;   // 90 communities
  struct Smem {
    Space<NT, kCells> s;
    Resident w;
  };
  static __device__ __forceinline__ Smem& mem() { return *reinterpret_cast<Smem*>(smem_raw); }
  static __device__ __forceinline__ Space<NT, kCells>& S() { return mem().s; }
  static __device__ __forceinline__ Resident& W() { return mem().w; }
};

enum { kModeCluster = 0, kModeGrid = 1 };

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Waits until *p reaches `goal`; false when the wait's limit has passed.
__device__ __forceinline__ bool wait_for(unsigned long long* p, unsigned long long goal, uint32_t* dead,
                                         unsigned long long limit_ns) {
  unsigned long long t0 = 0ull;
  for (unsigned spin = 0;; ++spin) {
    if (*reinterpret_cast<volatile unsigned long long*>(p) >= goal) return true;
    if ((spin & 1023u) != 1023u) continue;
    if (t0 == 0ull) t0 = now_ns();
    if (*reinterpret_cast<volatile uint32_t*>(dead) || now_ns() - t0 > limit_ns) {
      atomicOr(dead, 1u);
      return false;
    }
  }
}

// The blocks working on a level: K of the job's, this one `rank`.
template <typename X>
struct Team {
  int K_, rank_, mode;
  __device__ __forceinline__ int K() const { return X::kResident ? 1 : K_; }
  __device__ __forceinline__ int rank() const { return X::kResident ? 0 : rank_; }
  __device__ __forceinline__ int gt() const { return rank() * X::NT + (int)threadIdx.x; }
  __device__ __forceinline__ int stride() const { return K() * X::NT; }
  __device__ __forceinline__ bool lead() const { return rank() == 0 && threadIdx.x == 0; }
  // Barrier of the team's threads; global writes before it are seen after it.
  // A cluster uses the hardware barrier (release and acquire at cluster
  // scope).  A cooperative grid counts arrivals in device memory; its wait is
  // bounded, and false (in every thread of the block) ends the kernel.
  __device__ __forceinline__ bool sync() const {
    if (K() == 1) {
      __syncthreads();
      return true;
    }
    if (mode == kModeCluster) {
      cg::this_cluster().sync();
      return true;
    }
    return grid_sync(K_);
  }
  static __device__ __noinline__ bool grid_sync(int K) {
    __syncthreads();
    if constexpr (!X::kResident) {
      if (threadIdx.x == 0) {
        Ctl* c = X::W().ctl;
        X::S().goal += (unsigned long long)K;
        __threadfence();
        atomicAdd(&c->arrived, 1ull);
        X::S().alive = wait_for(&c->arrived, X::S().goal, &c->dead, X::S().wait_ns) ? 1 : 0;
        __threadfence();
      }
    }
    __syncthreads();
    return X::S().alive != 0;
  }
};

template <typename X>
__device__ __forceinline__ uint32_t block_excl(uint32_t v, uint32_t* total) {
  uint32_t* wtot = X::S().wtot;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t inc = warp_inclusive_scan(v);
  if (lane == 31) wtot[w] = inc;
  __syncthreads();
  if (w == 0) {
    uint32_t x = lane < X::NT / 32 ? wtot[lane] : 0u;
    x = warp_inclusive_scan(x);
    if (lane < X::NT / 32) wtot[lane] = x;
  }
  __syncthreads();
  const uint32_t base = w > 0 ? wtot[w - 1] : 0u;
  *total = wtot[X::NT / 32 - 1];
  __syncthreads();
  return base + inc - v;
}

// block_tree256 of the block's first 256 threads; the result in thread 0.
template <typename X>
__device__ __forceinline__ double first_tree(double s) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (w < 8) {
    for (int o = 16; o >= 1; o >>= 1) s = __dadd_rn(s, __shfl_down_sync(full, s, o));
    if (lane == 0) X::S().ws[w] = s;
  }
  __syncthreads();
  double r = 0.0;
  if (w == 0) {
    r = lane < 8 ? X::S().ws[lane] : 0.0;
    for (int o = 16; o >= 1; o >>= 1) r = __dadd_rn(r, __shfl_down_sync(full, r, o));
  }
  __syncthreads();
  return r;
}

// Group partials of the fixed-tree sum of val(load(i)), i < n (groups of
// 2048, a block each).  Both are called once per index, the loads of two
// indices before the first val, which may write.
template <typename X, typename G, typename F>
__device__ __forceinline__ void group_partials(const Team<X> T, int64_t n, double* partials, G load, F val) {
  constexpr int kPer = kGroup / X::NT;
  const int tid = threadIdx.x;
  double* stage = X::S().u.stage;
  const int64_t ng = max((int64_t)1, (n + kGroup - 1) / kGroup);
#pragma unroll 1
  for (int64_t g = T.rank(); g < ng; g += T.K()) {
    const int64_t i0 = g * kGroup + tid;
#pragma unroll 1
    for (int j = 0; j < kPer; j += 2) {
      const int64_t ia = i0 + j * X::NT, ib = ia + X::NT;
      decltype(load(ia)) xa, xb;
      if (ia < n) xa = load(ia);
      if (ib < n) xb = load(ib);
      stage[j * X::NT + tid] = ia < n ? val(ia, xa) : 0.0;
      stage[(j + 1) * X::NT + tid] = ib < n ? val(ib, xb) : 0.0;
    }
    __syncthreads();
    double s = 0.0;
    if (tid < 256) {
#pragma unroll
      for (int j = 0; j < 8; ++j) s = __dadd_rn(s, stage[j * 256 + tid]);
    }
    s = first_tree<X>(s);
    if (tid == 0) partials[g] = s;
  }
}

// Sum of the partials of n values, in every thread (at most 2048 partials).
template <typename X>
__device__ __forceinline__ double finish_sum(const double* partials, int64_t n) {
  if (n <= kGroup) return partials[0];   // the tree of one value
  const int64_t np = (n + kGroup - 1) / kGroup;
  double s = 0.0;
  if (threadIdx.x < 256) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int64_t i = j * 256 + (int)threadIdx.x;
      if (i < np) s = __dadd_rn(s, partials[i]);
    }
  }
  s = first_tree<X>(s);
  if (threadIdx.x == 0) X::S().bcast = s;
  __syncthreads();
  const double x = X::S().bcast;
  __syncthreads();
  return x;
}

// The block's share of the rows: those starting in its share of the entries
// and rows together (by entries alone, one block of 30 could own 100,000 empty
// rows: .3 ms a pass).  row0 and row1 become the first rows starting at or
// after the share's ends.
template <typename X>
__device__ __forceinline__ void find_rows(const Team<X> T, int32_t V, int64_t E) {
  auto& S = X::S();
  const int64_t x0 = (E + V) * T.rank() / T.K(), x1 = (E + V) * (T.rank() + 1) / T.K();
  if (threadIdx.x == 0) {   // a share that starts or ends at 0 does so at row 0
    S.row0 = 0;
    S.row1 = T.K() == 1 ? V : 0;
  }
  __syncthreads();
  if (T.K() > 1) {
    const int32_t* roff = X::W().roff;
#pragma unroll 2
    for (int32_t v = 1 + (int)threadIdx.x; v <= V; v += X::NT) {
      const int64_t a = (int64_t)roff[v - 1] + v - 1, b = (int64_t)roff[v] + v;
      if (T.rank() > 0 && a < x0 && b >= x0) S.row0 = v;
      if (a < x1 && b >= x1) S.row1 = v;
    }
    __syncthreads();
  }
}

// Row starts of a list of fewer than two entries a row, each row looking for
// its own: its gaps may be many and long.
template <typename X>
__device__ __forceinline__ void search_starts(const Team<X> T, const int32_t* src, int64_t E, int32_t V) {
  int32_t* roff = X::W().roff;
#pragma unroll 1
  for (int32_t r = T.gt(); r <= V; r += T.stride()) {
    int32_t lo = 0, hi = (int32_t)E;
    while (lo < hi) {
      const int32_t mid = (lo + hi) >> 1;
      if (src[mid] < r) lo = mid + 1;
      else hi = mid;
    }
    roff[r] = lo;
  }
}

// Rows r0..r1 start at entry e: few of them by the thread that met them, many
// by its block (long_gaps).  A coarse list ends in a gap of all vertices
// without edges: 189,000 written by one thread took 5.2 ms a level.
template <typename X>
__device__ __forceinline__ void row_starts(int32_t r0, int32_t r1, int32_t e) {
  auto& S = X::S();
  if constexpr (!X::kResident) {
    if (r1 - r0 >= 64) {
      const int p = atomicAdd(&S.ngap, 1);
      if (p < kGaps) {
        S.gap[p] = make_int4(r0, r1, e, 0);
        return;
      }
    }
  }
  int32_t* roff = X::W().roff;
#pragma unroll 1
  for (int32_t r = r0; r <= r1; ++r) roff[r] = e;
}

template <typename X>
__device__ __forceinline__ void long_gaps() {
  auto& S = X::S();
  int32_t* roff = X::W().roff;
  __syncthreads();
  const int n = min(S.ngap, kGaps);
#pragma unroll 1
  for (int g = 0; g < n; ++g) {
    const int4 x = S.gap[g];
#pragma unroll 2
    for (int32_t r = x.x + (int)threadIdx.x; r <= x.y; r += X::NT) roff[r] = x.z;
  }
}

// The decision for one vertex (apply_decision_kl of the level kernels).
// `last`: the pass ends the level, whose totals then stay as they are.
template <typename X, bool SINGLETON>
__device__ __forceinline__ void decide(int32_t i, int32_t own, int32_t bc, double bw, int32_t nseg, bool last) {
  auto& W = X::W();
  const int32_t raw = bc == kNone ? own : bc;
  const int32_t so = SINGLETON ? 1 : W.size[own], sb = SINGLETON ? 1 : W.size[raw];
  int32_t best = raw;
  if (so == 1 && sb == 1 && raw > own) best = own;
  W.next[i] = best;
  W.cand[i] = (so == 1 && nseg == 1 && raw != own && own < raw) ? raw : -1;
  if (best != own && !last) move_deltas<SINGLETON>(W.delta, own, best, W.k[i], __dadd_rn(bw, (double)W.loopw[i]));
}

// Rows [v0, v0 + return value) of the next tile: at most `cap` entries and a
// row a thread.  Uniform over the block.
template <typename X>
__device__ __forceinline__ int tile_rows(const int32_t* roff, int32_t v0, int32_t vend, int cap) {
  static_assert(Tile<X::NT>::kRows == X::NT, "a thread a row");
  const int32_t base = roff[v0];
  const int32_t v = v0 + 1 + (int)threadIdx.x;
  return __syncthreads_count(v <= vend && roff[v] - base <= cap);
}

// A list's rows: those of a symmetric list as it is (self loops among them,
// each entry standing for itself and its mirror), or of a merged CSR.
struct List {
  const int32_t* src;
  const int32_t* dst;
  const float* w;
  float copies;              // of an entry in the merged doubled list: 2, or 1 once merged
  __device__ __forceinline__ int32_t loop_apart(int32_t hasl) const { return copies == 1.0f ? hasl : 0; }
};

// Weight of a row's entry in the merged doubled list.
__device__ __forceinline__ double merged_w(const List& L, float w) { return (double)__fmul_rn(w, L.copies); }

// The block's best candidate from each thread's, in thread 0.
template <typename X>
__device__ __forceinline__ void block_best(double& g, int32_t& c, double& w) {
  auto& S = X::S();
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const double g2 = __shfl_xor_sync(full, g, o), w2 = __shfl_xor_sync(full, w, o);
    const int32_t c2 = __shfl_xor_sync(full, c, o);
    if (better(g2, c2, g, c)) { g = g2; c = c2; w = w2; }
  }
  if (lane == 0) { S.rg[wid] = g; S.rc[wid] = c; S.rw[wid] = w; }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 1; k < X::NT / 32; ++k)
      if (better(S.rg[k], S.rc[k], g, c)) { g = S.rg[k]; c = S.rc[k]; w = S.rw[k]; }
  __syncthreads();
}

// A row longer than a tile, in the first pass: the block strides over it.
template <typename X>
__device__ __noinline__ void long_first(const List L, int32_t v, bool last_pass) {
  auto& W = X::W();
  const int32_t beg = W.roff[v], end = W.roff[v + 1];
  const double kf = W.kfrac[v];
  double bg = 0.0, bw = 0.0;
  int32_t bc = kNone;
#pragma unroll 4
  for (int32_t e = beg + (int)threadIdx.x; e < end; e += X::NT) {
    const int32_t c = L.dst[e];
    const double w = merged_w(L, L.w[e]);
    const double g = __dsub_rn(w, __dmul_rn(W.k[c], kf));
    if (c != v && w != 0.0 && g > 0.0 && better(g, c, bg, bc)) { bg = g; bc = c; bw = w; }
  }
  block_best<X>(bg, bc, bw);
  if (threadIdx.x == 0) decide<X, true>(v, v, bc, bw, end - beg + L.loop_apart(W.hasl[v]), last_pass);
}

// First pass of a level: every neighbour is its own candidate.  Returns the
// first row longer than a tile, else vend.
template <typename X>
__device__ __forceinline__ int32_t moves_first_body(const List L, int32_t v, int32_t vend, bool last_pass) {
  constexpr int NT = X::NT;
  auto& S = X::S();
  auto& W = X::W();
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x;
#pragma unroll 1
  while (v < vend) {
    const int nv = tile_rows<X>(W.roff, v, vend, Tile<NT>::kInt);
    if (nv == 0) return v;
    const int32_t base = W.roff[v];
    const int n = W.roff[v + nv] - base;
    if (n > 0) {
      if (tid < nv) {
        S.kf[tid] = W.kfrac[v + tid];
        S.besth[tid] = S.bestl[tid] = 0u;
        S.bestc[tid] = kNone;
      }
      int jj[kItems], cc[kItems];
      double gg[kItems], wd[kItems];
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        const int x = q * NT + tid;
        jj[q] = -1;
        cc[q] = 0;
        wd[q] = 0.0;
        if (x < n) {
          jj[q] = L.src[base + x] - v;
          cc[q] = L.dst[base + x];
          wd[q] = merged_w(L, L.w[base + x]);
        }
      }
#pragma unroll
      for (int q = 0; q < kItems; ++q) gg[q] = jj[q] >= 0 ? W.k[cc[q]] : 0.0;   // singleton tot = k
      __syncthreads();
      unsigned last = 0;
      double pg[kItems];
      int32_t pc[kItems];
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        pg[q] = 0.0;
        pc[q] = kNone;
        if (q * NT + (tid & ~31) >= n) continue;   // whole warps
        const int j = jj[q];
        double g = 0.0;
        int32_t c = kNone;
        if (j >= 0 && cc[q] != v + j && wd[q] != 0.0) {                    // OneLevelKernel.cu:303
          const double t = __dsub_rn(wd[q], __dmul_rn(gg[q], S.kf[j]));    // OneLevelKernel.cu:307-313
          if (t > 0.0) { g = t; c = cc[q]; }
        }
        gg[q] = g;
        bool run_last;
        const int depth = run_depth(j, run_last);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {   // best candidate of the lane's row piece so far
          const double g2 = __shfl_up_sync(full, g, o);
          const int32_t c2 = __shfl_up_sync(full, c, o);
          if (o <= depth && better(g2, c2, g, c)) { g = g2; c = c2; }
        }
        if (j >= 0 && c != kNone && run_last) {
          last |= 1u << q;
          atomicMax(&S.besth[j], gain_hi(g));
        }
        pg[q] = g;
        pc[q] = c;
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q)
        if ((last >> q) & 1u) {
          if (gain_hi(pg[q]) == S.besth[jj[q]]) atomicMax(&S.bestl[jj[q]], gain_lo(pg[q]));
          else last &= ~(1u << q);
        }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q)
        if (((last >> q) & 1u) && gain_lo(pg[q]) == S.bestl[jj[q]]) atomicMin(&S.bestc[jj[q]], pc[q]);
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q)   // the winner's own entry
        if (jj[q] >= 0 && gg[q] > 0.0 && cc[q] == S.bestc[jj[q]]) S.bestw[jj[q]] = wd[q];
      __syncthreads();
      if (tid < nv) {
        const int32_t i = v + tid, len = W.roff[i + 1] - W.roff[i];
        const int32_t c = S.bestc[tid];
        // distinct candidates: one per neighbour, and the own community with a self loop
        if (len > 0)
          decide<X, true>(i, i, c, c == kNone ? 0.0 : S.bestw[tid], len + L.loop_apart(W.hasl[i]), last_pass);
      }
      __syncthreads();
    }
    v += nv;
  }
  return vend;
}

// (row, community) tables.  Integral weights: a 32-bit key (row << 18 |
// community, all ones when empty) and a 32-bit sum, both with the atomics
// shared memory has in hardware (64-bit adds and maxima are compare-and-swap
// loops there, which contend on the rows' favourite communities).
template <int NT, bool INT>
struct Table {
  static constexpr int kSlots = Tile<NT>::kSlots;
  static constexpr int kUsed = kSlots;
  static constexpr int kTile = Tile<NT>::kInt;
  static constexpr uint32_t kNoKey = 0xffffffffu;
  static __device__ __forceinline__ uint32_t* key_of(unsigned long long* slot) {
    return reinterpret_cast<uint32_t*>(slot);
  }
  static __device__ __forceinline__ uint32_t* sum_of(unsigned long long* slot) { return key_of(slot) + kSlots; }
  static __device__ __forceinline__ void insert(unsigned long long* slot, int32_t* ncl, uint16_t* claimed, int j,
                                                int32_t c, double w) {
    uint32_t *keys = key_of(slot), *sums = sum_of(slot);
    const uint32_t key = ((uint32_t)j << kCommBits) | (uint32_t)c;
    uint32_t h = (uint32_t)(((unsigned long long)key * 0x9E3779B97F4A7C15ull) >> (64 - Tile<NT>::kLog));
    for (int p = 0; p < kSlots; ++p) {   // a tile takes at most half the slots
      uint32_t cur = *reinterpret_cast<volatile uint32_t*>(&keys[h]);
      if (cur == kNoKey) {
        cur = atomicCAS(&keys[h], kNoKey, key);
        if (cur == kNoKey) {
          claimed[atomicAdd(ncl, 1)] = (uint16_t)h;
          cur = key;
        }
      }
      if (cur == key) { atomicAdd(&sums[h], (uint32_t)w); return; }
      h = (h + 1) & (kSlots - 1);
    }
  }
  static __device__ __forceinline__ void get(unsigned long long* slot, int s, int& j, int32_t& c, double& w) {
    const uint32_t key = key_of(slot)[s];
    j = (int)(key >> kCommBits);
    c = (int32_t)(key & ((1u << kCommBits) - 1u));
    w = (double)sum_of(slot)[s];
  }
  static __device__ __forceinline__ void clear(unsigned long long* slot, int s) {
    key_of(slot)[s] = kNoKey;
    sum_of(slot)[s] = 0u;
  }
};
static_assert(kCommBits + 10 < 32, "no key is all ones");

template <int NT>
struct Table<NT, false> {
  static constexpr int kTile = Tile<NT>::kF64;
  static constexpr int kHalf = Tile<NT>::kSlots / 2;   // keys below, FP64 sums above
  static constexpr int kUsed = kHalf;
  static __device__ __forceinline__ void insert(unsigned long long* slot, int32_t* ncl, uint16_t* claimed, int j,
                                                int32_t c, double w) {
    const unsigned long long key = ((unsigned long long)j << 32) | (uint32_t)c;
    double* sum = reinterpret_cast<double*>(slot + kHalf);
    uint32_t h = (uint32_t)((key * 0x9E3779B97F4A7C15ull) >> (64 - Tile<NT>::kLog + 1));
    for (int p = 0; p < kHalf; ++p) {
      const unsigned long long prev = atomicCAS(&slot[h], kEmpty, key);
      if (prev == kEmpty) claimed[atomicAdd(ncl, 1)] = (uint16_t)h;
      if (prev == kEmpty || prev == key) { atomicAdd(&sum[h], w); return; }
      h = (h + 1) & (kHalf - 1);
    }
  }
  static __device__ __forceinline__ void get(unsigned long long* slot, int s, int& j, int32_t& c, double& w) {
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

// Rows longer than a tile, in a later pass.  Each has a table of its own in
// device memory, twice as many slots as entries (keys over key[0], FP64 sums
// over key[1] and wsum, which the sort does not need meanwhile), so that the
// whole team works on it: a block reads the entries of long rows within its
// share of the list, adds them up in shared memory a tile at a time, and adds
// each tile's communities to the row's table (hub_insert); then a block per
// row takes the best and leaves the table empty (hub_pick).  One block alone,
// hashing a row of 60,000 entries part by part in shared memory, took 1 ms a
// pass with integral weights and 7 with others.
template <typename X>
struct HubTable {
  int32_t* key;
  double* sum;
  uint32_t slots;
  __device__ __forceinline__ explicit HubTable(int32_t v) {
    auto& W = X::W();
    const int64_t beg = W.roff[v];
    key = (int32_t*)W.key[0] + 2 * beg;
    sum = (double*)W.key[1] + 2 * beg;
    slots = 2u * (uint32_t)(W.roff[v + 1] - beg);
  }
};

template <typename X>
__device__ __noinline__ void hub_clear(const Team<X> T) {
  auto& W = X::W();
  const int n = (int)W.ctl->nlong;
#pragma unroll 1
  for (int i = T.rank(); i < n; i += T.K()) {
    const HubTable<X> H(W.longs[i]);
#pragma unroll 4
    for (uint32_t x = threadIdx.x; x < H.slots; x += X::NT) {
      H.key[x] = kNone;
      H.sum[x] = 0.0;
    }
  }
}

// (Behind moves_hash, which leaves its table empty.)
template <typename X, bool INT>
__device__ __noinline__ void hub_insert(const Team<X> T, const List L, int64_t E) {
  using Tab = Table<X::NT, INT>;
  auto& S = X::S();
  auto& W = X::W();
  unsigned long long* slot = S.u.slot;
  const int tid = threadIdx.x;
  const int n = (int)W.ctl->nlong;
  const int32_t x0 = (int32_t)(E * T.rank() / T.K()), x1 = (int32_t)(E * (T.rank() + 1) / T.K());
#pragma unroll 1
  for (int i0 = 0; i0 < n; i0 += X::NT) {
    const int32_t v = i0 + tid < n ? W.longs[i0 + tid] : -1;
    bool mine = false;
    if (v >= 0) {
      const int32_t beg = W.roff[v], end = W.roff[v + 1];
      mine = end - beg > Tab::kTile && beg < x1 && end > x0;
    }
    for (;;) {   // a few of the rows at a time
      if (tid == 0) S.nhub = 0;
      __syncthreads();
      if (mine) {
        const int p = atomicAdd(&S.nhub, 1);
        if (p < kHubs) {
          S.hub[p] = v;
          mine = false;
        }
      }
      __syncthreads();
      const int found = min(S.nhub, kHubs);
#pragma unroll 1
      for (int h = 0; h < found; ++h) {
        const int32_t row = S.hub[h];
        const HubTable<X> H(row);
        const int32_t lo = max(W.roff[row], x0), hi = min(W.roff[row + 1], x1);
#pragma unroll 1
        for (int32_t e0 = lo; e0 < hi; e0 += Tab::kTile) {
#pragma unroll 4
          for (int q = 0; q < Tab::kTile / X::NT; ++q) {
            const int32_t e = e0 + q * X::NT + tid;
            if (e < hi) {
              const int32_t d = L.dst[e];
              if (d != row) Tab::insert(slot, &S.nclaimed, S.claimed, 0, W.comm[d], merged_w(L, L.w[e]));
            }
          }
          __syncthreads();
          const int nc = S.nclaimed;
#pragma unroll 1
          for (int x = tid; x < nc; x += X::NT) {
            int j;
            int32_t c;
            double w;
            Tab::get(slot, S.claimed[x], j, c, w);
            Tab::clear(slot, S.claimed[x]);
            uint32_t at = (uint32_t)(((uint64_t)((uint32_t)c * 0x9E3779B1u) * H.slots) >> 32);
            for (uint32_t p = 0; p < H.slots; ++p) {   // at most half are ever taken
              const int32_t cur = atomicCAS(&H.key[at], kNone, c);
              if (cur == kNone || cur == c) {
                atomicAdd(&H.sum[at], w);
                break;
              }
              if (++at == H.slots) at = 0;
            }
          }
          __syncthreads();
          if (tid == 0) S.nclaimed = 0;
          __syncthreads();
        }
      }
      if (!__syncthreads_or(mine)) break;
    }
  }
}

template <typename X, bool INT>
__device__ __noinline__ void hub_pick(const Team<X> T, bool last_pass) {
  auto& S = X::S();
  auto& W = X::W();
  const int n = (int)W.ctl->nlong;
#pragma unroll 1
  for (int i = T.rank(); i < n; i += T.K()) {
    const int32_t v = W.longs[i];
    const HubTable<X> H(v);
    if (H.slots <= 2u * Table<X::NT, INT>::kTile) continue;
    if (threadIdx.x == 0) S.nhub = 0;
    __syncthreads();
    const double kf = W.kfrac[v];
    const int32_t own = W.comm[v];
    double bg = 0.0, bw = 0.0;
    int32_t bc = kNone;
    uint32_t met = 0;   // communities, and bit 31: the row's own
#pragma unroll 4
    for (uint32_t x = threadIdx.x; x < H.slots; x += X::NT) {
      const int32_t c = H.key[x];
      if (c == kNone) continue;
      const double w = H.sum[x];
      H.key[x] = kNone;
      H.sum[x] = 0.0;
      met = (met + 1) | (c == own ? 1u << 31 : 0u);
      if (w != 0.0) {
        const double g = __dsub_rn(w, __dmul_rn(W.tot[c], kf));
        if (g > 0.0 && better(g, c, bg, bc)) { bg = g; bc = c; bw = w; }
      }
    }
    const uint32_t many = __reduce_add_sync(0xffffffffu, met & 0x7fffffffu);
    const uint32_t own_met = __reduce_or_sync(0xffffffffu, met & (1u << 31));
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&S.nhub, (int)many);
      if (own_met) atomicOr(&S.nhub, 1 << 30);   // (sums stay far below)
    }
    block_best<X>(bg, bc, bw);   // (its barriers order nhub too)
    if (threadIdx.x == 0) {
      const int32_t s = S.nhub;
      const int32_t nseg = (s & ((1 << 30) - 1)) + ((W.hasl[v] && !(s >> 30)) ? 1 : 0);
      decide<X, false>(v, own, bc, bw, nseg, last_pass);
    }
    __syncthreads();
  }
}

// A later pass: rows hashed tile by tile.  Returns as moves_first_body.
template <typename X, bool INT>
__device__ __forceinline__ int32_t moves_hash_body(const List L, int32_t v, int32_t vend, bool last_pass) {
  constexpr int NT = X::NT;
  using Tab = Table<NT, INT>;
  constexpr int kItems = Tab::kTile / NT;
  auto& S = X::S();
  auto& W = X::W();
  const int tid = threadIdx.x;
  unsigned long long* slot = S.u.slot;
#pragma unroll 2
  for (int s = tid; s < Tab::kUsed; s += NT) Tab::clear(slot, s);
  if (tid == 0) S.nclaimed = 0;
  __syncthreads();
#pragma unroll 1
  while (v < vend) {
    const int nv = tile_rows<X>(W.roff, v, vend, Tab::kTile);
    if (nv == 0) return v;
    const int32_t base = W.roff[v];
    const int n = W.roff[v + nv] - base;
    if (n > 0) {
      if (tid < nv) {
        S.own[tid] = W.comm[v + tid];
        S.kf[tid] = W.kfrac[v + tid];
        S.besth[tid] = S.bestl[tid] = 0u;
        S.bestc[tid] = kNone;
        S.nseg[tid] = 0;
      }
      int jj[kItems];
      int32_t cc[kItems];
      double wd[kItems];
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        const int x = q * NT + tid;
        jj[q] = -1;
        cc[q] = 0;
        wd[q] = 0.0;
        if (x < n) {
          const int32_t u = L.src[base + x], d = L.dst[base + x];
          if (u != d) jj[q] = u - v;
          cc[q] = d;
          wd[q] = merged_w(L, L.w[base + x]);
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
        const int x = q * NT + tid;
        gg[q] = 0.0;
        jj[q] = -1;
        if (x < nc) {
          const int sl = S.claimed[x];
          Tab::get(slot, sl, jj[q], cc[q], wd[q]);
          Tab::clear(slot, sl);
        }
      }
#pragma unroll
      for (int q = 0; q < kItems; ++q)
        if (jj[q] >= 0 && wd[q] != 0.0) gg[q] = W.tot[cc[q]];
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        if (jj[q] >= 0) {
          atomicAdd(&S.nseg[jj[q]], 1);
          if (wd[q] != 0.0) gg[q] = __dsub_rn(wd[q], __dmul_rn(gg[q], S.kf[jj[q]]));
          if (gg[q] > 0.0) atomicMax(&S.besth[jj[q]], gain_hi(gg[q]));
        }
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q)
        if (jj[q] >= 0 && gg[q] > 0.0) {
          if (gain_hi(gg[q]) == S.besth[jj[q]]) atomicMax(&S.bestl[jj[q]], gain_lo(gg[q]));
          else gg[q] = 0.0;
        }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q)         // smallest community among the best gains
        if (jj[q] >= 0 && gg[q] > 0.0 && gain_lo(gg[q]) == S.bestl[jj[q]]) atomicMin(&S.bestc[jj[q]], cc[q]);
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q)
        if (jj[q] >= 0 && cc[q] == S.bestc[jj[q]]) S.bestw[jj[q]] = wd[q];
      if (tid == 0) S.nclaimed = 0;
      __syncthreads();
      if (tid < nv) {
        const int32_t i = v + tid;
        if (W.roff[i + 1] > W.roff[i]) {
          const int32_t c = S.bestc[tid], s = S.nseg[tid];
          const int32_t nseg = (s & ((1 << 30) - 1)) + ((W.hasl[i] && !(s >> 30)) ? 1 : 0);
          decide<X, false>(i, S.own[tid], c, c == kNone ? 0.0 : S.bestw[tid], nseg, last_pass);
        }
      }
      __syncthreads();
    }
    v += nv;
  }
  return vend;
}

// Over device memory: out of line, where registers are short, with the long
// rows between (inside the tiles' loops they cost every graph 2-3 %).  A level
// in shared memory has no row longer than a tile.
template <typename X>
__device__ __noinline__ int32_t moves_first_call(const List L, int32_t v, int32_t vend, bool last) {
  return moves_first_body<X>(L, v, vend, last);
}
template <typename X, bool INT>
__device__ __noinline__ int32_t moves_hash_call(const List L, int32_t v, int32_t vend, bool last) {
  return moves_hash_body<X, INT>(L, v, vend, last);
}
template <typename X>
__device__ __forceinline__ void moves_first(const List L, int32_t v, int32_t vend, bool last) {
  if constexpr (X::kResident) {
    moves_first_body<X>(L, v, vend, last);
  } else {
#pragma unroll 1
    while ((v = moves_first_call<X>(L, v, vend, last)) < vend) long_first<X>(L, v++, last);
  }
}
template <typename X, bool INT>
__device__ __forceinline__ void moves_hash(const List L, int32_t v, int32_t vend, bool last) {
  if constexpr (X::kResident && INT) {
    moves_hash_body<X, INT>(L, v, vend, last);
  } else {
#pragma unroll 1
    while ((v = moves_hash_call<X, INT>(L, v, vend, last)) < vend) ++v;   // hub_insert's
  }
}

struct Committed {
  Delta d;
  double tot, in, k;
  int32_t size, next;
};

// Commit of a pass (communitySetKernel) with the Q partials of the new state.
// FINAL: the level's last commit, which also takes every community's smallest
// member.
template <typename X, bool FINAL>
__device__ __forceinline__ void commit(const Team<X> T, int32_t V, double m) {
  auto& W = X::W();
  const double twom = __dmul_rn(2.0, m);
  group_partials<X>(
      T, V, W.qpart,
      [&](int64_t c) {
        return Committed{W.delta[c], W.tot[c], W.in[c], W.k[c], W.size[c], W.next[c]};
      },
      [&](int64_t c, Committed& x) {
        delta_commit(x.d, x.k, x.tot, x.in, x.size);
        W.comm[c] = x.next;
        if (FINAL) {
          atomicMin(&W.minidx[x.next], (int32_t)c);
        } else {
          W.delta[c] = x.d;
          W.tot[c] = x.tot;
          W.in[c] = x.in;
          W.size[c] = x.size;
        }
        return q_term(x.in, x.tot, m, twom);
      });
}

// The state behind the level's last commit, which left its totals where they
// were: for the calls that follow a run (its labels go with the partitions).
template <typename X>
__device__ __noinline__ void keep_state(const Team<X> T, int32_t V, double* state) {
  auto& W = X::W();
  double *tot = state, *in = state + V;
  int32_t* size = reinterpret_cast<int32_t*>(in + V);
#pragma unroll 1
  for (int32_t c = T.gt(); c < V; c += T.stride()) {
    Committed x{W.delta[c], W.tot[c], W.in[c], W.k[c], W.size[c], 0};
    delta_commit(x.d, x.k, x.tot, x.in, x.size);
    tot[c] = x.tot;
    in[c] = x.in;
    size[c] = x.size;
  }
}

// Entries of the list checked: ids and weights, strict order, and symmetry by
// order-free fingerprints: two 64-bit hashes of (src, dst, weight bits) summed
// mod 2^64 against those of (dst, src, weight bits).
template <typename X>
__device__ __noinline__ void check_list(const Team<X> T, const List L, int64_t E, int32_t V) {
  const uint64_t K1 = 0x243F6A8885A308D3ull, K2 = 0x13198A2E03707344ull;
  const unsigned full = 0xffffffffu;
  uint64_t d1 = 0, d2 = 0;
  uint32_t f = 0;
#pragma unroll 1
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
  if ((threadIdx.x & 31) == 0) {
    Ctl* c = X::W().ctl;
    if (d1) atomicAdd(&c->sums[0], (unsigned long long)d1);
    if (d2) atomicAdd(&c->sums[1], (unsigned long long)d2);
    if (f) atomicOr(&c->check, f);
  }
}

// A resident level's coarse list is summed pair by pair in shared memory.
template <typename X>
__device__ __forceinline__ bool cells_fit(int32_t C) {
  return X::kResident && C <= 1024 && C * C <= X::kCells;
}

// Keys with their values: 32-bit keys side by side with them, one scattered
// store of 8 bytes each a pass instead of two of 4 (coarsening 1.9 M entries:
// 275 us before, 237 now).
template <typename Key>
struct Keyed {
  uint64_t* key;
  float* val;
  static constexpr bool kPair = sizeof(Key) == 4;
  __device__ __forceinline__ Key at(int64_t i) const {
    if constexpr (kPair) return reinterpret_cast<const uint2*>(key)[i].x;
    else return key[i];
  }
  __device__ __forceinline__ void get(int64_t i, Key& k, float& x) const {
    if constexpr (kPair) {
      const uint2 p = reinterpret_cast<const uint2*>(key)[i];
      k = p.x;
      x = __uint_as_float(p.y);
    } else {
      k = key[i];
      x = val[i];
    }
  }
  __device__ __forceinline__ void put(int64_t i, Key k, float x) const {
    if constexpr (kPair) {
      reinterpret_cast<uint2*>(key)[i] = make_uint2(k, __float_as_uint(x));
    } else {
      key[i] = k;
      val[i] = x;
    }
  }
};

// Stable LSD sort over the team of n keys by their low `bits` bits, made with
// their values by gen(i, key, val): block r owns the r-th share of the
// positions, counts its digits, and places its keys after those of all blocks
// before it.  Clears wsum.  Returns which of W.key / W.val holds the result
// (-1: a barrier's wait ran out).
template <typename X, typename Key, typename G>
__device__ __forceinline__ int sort_keys(const Team<X> T, int64_t n, int bits, G gen) {
  constexpr int NT = X::NT, kIt = 4, kQ = NT / kDigits;
  auto& S = X::S();
  auto& W = X::W();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int np = (bits + 7) / 8, width = (bits + np - 1) / np;
  const uint32_t dmask = (1u << width) - 1u;
  const int64_t s0 = n * T.rank() / T.K(), s1 = n * (T.rank() + 1) / T.K();
  int cur = 0;
#pragma unroll 1
  for (int p = 0; p < np; ++p) {
    const Keyed<Key> from{W.key[cur], W.val[cur]}, to{W.key[cur ^ 1], W.val[cur ^ 1]};
    if (tid < kDigits) S.hist[tid] = 0;
    __syncthreads();
    if (p == 0) {
      double* wsum = W.wsum;
#pragma unroll 4
      for (int x = tid; x < (NT / 32) * kDigits; x += NT) (&S.u.sort.meet[0][0])[x] = 0;
#pragma unroll 2
      for (int64_t e = s0 + tid; e < s1; e += NT) {
        Key key;
        float x;
        gen(e, key, x);
        from.put(e, key, x);
        wsum[e] = 0.0;
        atomicAdd(&S.hist[(uint32_t)key & dmask], 1u);
      }
    } else {
#pragma unroll 4
      for (int64_t e = s0 + tid; e < s1; e += NT)
        atomicAdd(&S.hist[(uint32_t)(from.at(e) >> (p * width)) & dmask], 1u);
    }
    __syncthreads();
    uint32_t tot = 0, pre = 0;
    if (T.K() > 1) {
      // digit counts of all blocks: kQ threads a digit, then their sums
      if (tid < kDigits) W.ghist[T.rank() * kDigits + tid] = S.hist[tid];
      if (!T.sync()) return -1;
      const int d = tid & (kDigits - 1), q = tid / kDigits;
      const int r0 = T.K() * q / kQ, r1 = T.K() * (q + 1) / kQ;
#pragma unroll 8
      for (int r = r0; r < r1; ++r) {
        const uint32_t c = W.ghist[r * kDigits + d];
        if (r < T.rank()) pre += c;
        tot += c;
      }
      S.u.part[0][q][d] = tot;
      S.u.part[1][q][d] = pre;
      __syncthreads();
      tot = pre = 0;
      if (tid < kDigits) {
#pragma unroll
        for (int k = 0; k < kQ; ++k) {
          tot += S.u.part[0][k][tid];
          pre += S.u.part[1][k][tid];
        }
      }
    } else if (tid < kDigits) {
      tot = S.hist[tid];
    }
    uint32_t all;
    const uint32_t ex = block_excl<X>(tot, &all);
    if (tid < kDigits) S.dbase[tid] = ex + pre;
#pragma unroll 1
    for (int64_t t0 = s0; t0 < s1; t0 += NT * kIt) {
#pragma unroll 2
      for (int x = tid; x < (NT / 32) * kDigits; x += NT) (&S.u.sort.wc[0][0])[x] = 0;
      Key key[kIt];
      uint32_t rank[kIt], dg[kIt];
      float val[kIt];
      const int64_t base = t0 + (int64_t)wid * 32 * kIt;
#pragma unroll
      for (int j = 0; j < kIt; ++j) {
        const int64_t i = base + j * 32 + lane;
        key[j] = Key(0);
        val[j] = 0.0f;
        if (i < s1) from.get(i, key[j], val[j]);
        dg[j] = i < s1 ? (uint32_t)(key[j] >> (p * width)) & dmask : (uint32_t)kDigits;
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < kIt; ++j) {
        // lanes of a digit meet in a shared word (with a match instruction
        // coarsening 1.9 M entries took 295 us instead of 275)
        const bool in = dg[j] < (uint32_t)kDigits;
        if (in) atomicOr(&S.u.sort.meet[wid][dg[j]], 1u << lane);
        __syncwarp();
        const unsigned peers = in ? S.u.sort.meet[wid][dg[j]] : 0u;
        const uint32_t before = in ? S.u.sort.wc[wid][dg[j]] : 0u;
        rank[j] = before + __popc(peers & lt);
        __syncwarp();
        if (in && (peers & lt) == 0) {
          S.u.sort.wc[wid][dg[j]] = before + __popc(peers);
          S.u.sort.meet[wid][dg[j]] = 0u;
        }
        __syncwarp();
      }
      __syncthreads();
      if (tid < kDigits) {
        uint32_t run = S.dbase[tid];
#pragma unroll 8
        for (int w = 0; w < NT / 32; ++w) {
          const uint32_t c = S.u.sort.wc[w][tid];
          S.u.sort.wc[w][tid] = run;
          run += c;
        }
        S.dbase[tid] = run;
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < kIt; ++j)
        if (dg[j] < (uint32_t)kDigits) {
          const uint32_t o = S.u.sort.wc[wid][dg[j]] + rank[j];
          to.put(o, key[j], val[j]);
        }
      __syncthreads();
    }
    if (!T.sync()) return -1;
    cur ^= 1;
  }
  return cur;
}

// Runs of equal keys that `counts` at their first entry: those started before
// the block's share, and all of them.  False: a barrier's wait ran out.
template <typename X, typename Key, typename P>
__device__ __forceinline__ bool count_runs(const Team<X> T, const Keyed<Key> key, int64_t s0, int64_t s1, uint32_t& run,
                                           uint32_t& cnt, P counts) {
  auto& W = X::W();
  uint32_t heads = 0;
#pragma unroll 1
  for (int64_t i0 = s0; i0 < s1; i0 += X::NT) {
    const int64_t i = i0 + threadIdx.x;
    const Key k = i < s1 ? key.at(i) : Key(0);
    heads += __syncthreads_count(i < s1 && (i == 0 || k != key.at(i - 1)) && counts(k));
  }
  run = 0;
  cnt = heads;
  if (T.K() > 1) {
    if (threadIdx.x == 0) W.ctl->count[1][T.rank()] = heads;
    if (!T.sync()) return false;
    cnt = 0;
#pragma unroll 4
    for (int r = 0; r < T.K(); ++r) {
      const uint32_t c = W.ctl->count[1][r];
      if (r < T.rank()) run += c;
      cnt += c;
    }
  }
  return true;
}

// The coarse list of a level of C communities (new ids W.newid of the labels
// W.comm) into (osrc, odst, ow); returns its length (-1: a barrier's wait ran
// out).  packed: whole weights and degrees below 2^30, so that a sum over the
// level stays far below 2^63 (a whole weight alone may be any float from 2^23
// up, and 2^64 fits no integer).
template <typename X, typename Key>
__device__ __noinline__ int64_t coarsen(const Team<X> T, const List L, int64_t E, int32_t C, bool packed,
                                        int32_t* osrc, int32_t* odst, float* ow) {
  constexpr int NT = X::NT, kIt = 4;
  auto& S = X::S();
  auto& W = X::W();
  const int tid = threadIdx.x;
  if (cells_fit<X>(C)) {
    // few communities, one block: a sum for every pair of them, the pairs met
    // (sums are positive: weight 0 counts 1) written in order, to the resident
    // list as well
    const int cells = C * C;
#pragma unroll 1
    for (int x = tid; x < cells; x += NT) S.u.cell[x] = 0.0;
    __syncthreads();
#pragma unroll 4
    for (int64_t e = tid; e < E; e += NT) {
      const float x = L.w[e];
      const int cell = W.newid[W.comm[L.src[e]]] * C + W.newid[W.comm[L.dst[e]]];
      // those add as integers (shared memory adds them in place)
      if (packed) atomicAdd(reinterpret_cast<unsigned long long*>(&S.u.cell[cell]),
                              x == 0.0f ? 1ull : (unsigned long long)x);       // InducedGraphKernel.cu:38-39
      else atomicAdd(&S.u.cell[cell], x == 0.0f ? 1.0 : (double)x);
    }
    __syncthreads();
    // a run of consecutive cells a thread
    const int per = (cells + NT - 1) / NT, x0 = min(tid * per, cells), x1 = min(x0 + per, cells);
    uint32_t met = 0;
#pragma unroll 4
    for (int x = x0; x < x1; ++x) met += S.u.cell[x] != 0.0 ? 1u : 0u;   // (an integer's bits are 0 for 0 alone)
    uint32_t all;
    uint32_t r = block_excl<X>(met, &all);
    int row = x0 / C, column = x0 % C;
    if constexpr (X::kResident) {
#pragma unroll 1
      for (int x = x0; x < x1; ++x) {
        const double sum = S.u.cell[x];
        if (sum != 0.0) {
          const float w = __double2float_rn(packed ? (double)__double_as_longlong(sum) : sum);
          W.src[r] = osrc[r] = row;
          W.dst[r] = odst[r] = column;
          W.w[r] = ow[r] = w;
          ++r;
        }
        if (++column == C) {
          column = 0;
          ++row;
        }
      }
    }
    __syncthreads();
    return (int64_t)all;
  }
  int b = 1;
  while ((1 << b) < C) ++b;
  const int32_t *comm = W.comm, *newid = W.newid;
  const int cur = sort_keys<X, Key>(T, E, 2 * b, [&](int64_t e, Key& k, float& x) {
    k = ((Key)newid[comm[L.src[e]]] << b) | (Key)newid[comm[L.dst[e]]];
    x = L.w[e];
    x = x == 0.0f ? 1.0f : x;       // InducedGraphKernel.cu:38-39
  });
  if (cur < 0) return -1;
  // runs of equal keys: heads counted per block, then each run's pieces added
  const Keyed<Key> key{W.key[cur], W.val[cur]};
  double* wsum = W.wsum;
  const int64_t s0 = E * T.rank() / T.K(), s1 = E * (T.rank() + 1) / T.K();
  uint32_t run, cnt;
  if (!count_runs<X>(T, key, s0, s1, run, cnt, [](Key) { return true; })) return -1;
  const Key cmask = (Key(1) << b) - 1;
#pragma unroll 1
  for (int64_t t0 = s0; t0 < s1; t0 += NT * kIt) {
    const int64_t i0 = t0 + (int64_t)tid * kIt;
    Key k[kIt + 1];
    float xs[kIt];
    uint32_t hm = 0;
    k[0] = i0 > 0 && i0 < s1 ? key.at(i0 - 1) : Key(0);
#pragma unroll
    for (int j = 0; j < kIt; ++j) {
      k[j + 1] = Key(0);
      if (i0 + j < s1) key.get(i0 + j, k[j + 1], xs[j]);
      if (i0 + j < s1 && (i0 + j == 0 || k[j + 1] != k[j])) hm |= 1u << j;
    }
    uint32_t all;
    uint32_t r = run + block_excl<X>((uint32_t)__popc(hm), &all);   // runs started before the thread
    run += all;
    double s = 0.0;
    bool any = false;
#pragma unroll
    for (int j = 0; j < kIt; ++j) {
      if (i0 + j < s1) {
        if ((hm >> j) & 1u) {
          if (any) atomicAdd(&wsum[r - 1], s);
          s = 0.0;
          osrc[r] = (int32_t)(k[j + 1] >> b);
          odst[r] = (int32_t)(k[j + 1] & cmask);
          ++r;
        }
        s = __dadd_rn(s, (double)xs[j]);
        any = true;
      }
    }
    if (any) atomicAdd(&wsum[r - 1], s);
  }
  if (!T.sync()) return -1;
#pragma unroll 2
  for (int64_t i = T.gt(); i < cnt; i += T.stride()) ow[i] = __double2float_rn(wsum[i]);
  if (!T.sync()) return -1;   // the next level's team may be smaller
  return (int64_t)cnt;
}

// CSR of a list that is not sorted and symmetric: the doubled list sorted by
// (src, dst), equal pairs merged, row by row in W.csrc / cdst / cw; degrees
// and self loops on the way (as csr_scan_kernel).  Returns the entries (-1: a
// barrier's wait ran out).
template <typename X, typename Key>
__device__ __noinline__ int64_t build_csr(const Team<X> T, const List L, int64_t E, int32_t V) {
  constexpr int NT = X::NT, kIt = 4;
  auto& W = X::W();
  int b = 1;
  while ((1 << b) < V) ++b;
  const int64_t n = 2 * E;
  const int cur = sort_keys<X, Key>(T, n, 2 * b, [&](int64_t e, Key& k, float& x) {
    const int64_t q = e < E ? e : e - E;
    const Key u = (Key)L.src[q], d = (Key)L.dst[q];
    k = e < E ? (u << b) | d : (d << b) | u;
    x = L.w[q];
  });
  if (cur < 0) return -1;
  const Keyed<Key> key{W.key[cur], W.val[cur]};
  double* wsum = W.wsum;
  const Key cmask = (Key(1) << b) - 1;
  const int64_t s0 = n * T.rank() / T.K(), s1 = n * (T.rank() + 1) / T.K();
  uint32_t run, cnt;
  if (!count_runs<X>(T, key, s0, s1, run, cnt, [&](Key k) { return (k >> b) != (k & cmask); })) return -1;
#pragma unroll 1
  for (int64_t t0 = s0; t0 < s1; t0 += NT * kIt) {
    const int64_t i0 = t0 + (int64_t)threadIdx.x * kIt;
    Key k[kIt + 2];
    float xs[kIt + 1];
    uint32_t hm = 0;
    k[0] = i0 > 0 && i0 < s1 ? key.at(i0 - 1) : Key(0);
#pragma unroll
    for (int j = 0; j <= kIt; ++j) {
      k[j + 1] = Key(0);
      if (i0 + j < n && i0 < s1) key.get(i0 + j, k[j + 1], xs[j]);
    }
#pragma unroll
    for (int j = 0; j < kIt; ++j)
      if (i0 + j < s1 && (i0 + j == 0 || k[j + 1] != k[j]) && (k[j + 1] >> b) != (k[j + 1] & cmask)) hm |= 1u << j;
    uint32_t all;
    uint32_t r = run + block_excl<X>((uint32_t)__popc(hm), &all);
    run += all;
    double s = 0.0, deg = 0.0;
    bool any = false;
#pragma unroll
    for (int j = 0; j < kIt; ++j) {
      const int64_t i = i0 + j;
      if (i < s1) {
        const int32_t u = (int32_t)(k[j + 1] >> b), d = (int32_t)(k[j + 1] & cmask);
        const float x = xs[j];
        if ((hm >> j) & 1u) {
          if (any) atomicAdd(&wsum[r - 1], s);
          s = 0.0;
          any = false;
          W.csrc[r] = u;
          W.cdst[r] = d;
          ++r;
        }
        if (u != d) {
          s = __dadd_rn(s, (double)x);
          any = true;
        } else if (i == n - 1 || k[j + 2] != k[j + 1]) {   // the last self-loop entry (InitKernel.cu:181-194)
          W.loopw[u] = x;
          W.hasl[u] = 1;
        }
        float f = x == 0.0f ? 1.0f : x;                    // InitKernel.cu:165-170
        if (u == d) f *= 2.0f;
        deg = __dadd_rn(deg, (double)f);
        if (j == kIt - 1 || i == s1 - 1 || (int32_t)(k[j + 2] >> b) != u) {
          atomicAdd(&W.k[u], deg);
          deg = 0.0;
        }
      }
    }
    if (any) atomicAdd(&wsum[r - 1], s);
  }
  if (!T.sync()) return -1;
#pragma unroll 2
  for (int64_t i = T.gt(); i < cnt; i += T.stride()) W.cw[i] = __double2float_rn(wsum[i]);
  if (!T.sync()) return -1;
  return (int64_t)cnt;
}

// Where a job's levels stand, the same in every thread of its team.
struct At {
  int32_t V;
  int64_t E;
  int32_t ncomms = 0;
  int buf = -1, nlev = 0, status = LVG_OK;
  bool open = false, symmetric = true, bad = false, tail = false, mid = false;
  bool any_order = false;   // the list may be other than sorted and symmetric, and there is room for that
  double mod = 0.0;
  int64_t part_off = 0;
};

struct Row {
  double k;
  float loopw;
  int32_t len;
};

// The level loop from `at` on, until the run has ended, a level is left open,
// or (not resident) a level fits one block's shared memory.  False: a
// barrier's wait ran out.
template <typename X>
__device__ __forceinline__ bool run_levels(Team<X>& T, const SmallCfg& cfg, At& at) {
  constexpr int NT = X::NT;
  auto& S = X::S();
  auto& W = X::W();
  const SmallJob& J = S.J;
  const bool lead = T.lead();
  List L{J.src, J.dst, J.w, 2.0f};
  if (at.buf >= 0) {
    int32_t *ls, *ld;
    float* lw;
    list_of(J.lists, J.E, at.buf, &ls, &ld, &lw);
    L = List{ls, ld, lw, 2.0f};
  }
  int64_t res_v = 0;
  bool list_here = false;   // the resident list is already this level's
  for (;;) {
    const long long t0 = clock64();
    const int level = J.level0 + at.nlev;
    const int32_t V = at.V;
    const int64_t E = at.E;
    if (at.nlev >= kSmallLevels || (J.parts && at.part_off + 2 * (int64_t)V > J.parts_cap)) { at.open = true; return true; }
    if (!X::kResident) {
      if (V <= kResV && E <= kResE && !at.any_order) { at.tail = true; return true; }
      // below this a cluster's barriers save more than the chip's width does
      // (a level of 117 Ki entries takes 154 us on the grid, 199 on a cluster;
      // one of 12 Ki 96 and 68; one of 2 Ki entries and 189,000 vertices 504
      // and 561: vertices count as entries do)
      if (T.mode == kModeGrid && E + V <= kSmallClusterEntries) { at.mid = true; return true; }
      // few entries for so many blocks: the last ones leave
      if (T.mode == kModeGrid && T.K_ > 1) {
        T.K_ = (int)min((int64_t)T.K_, (E + V + kGridEntries - 1) / kGridEntries);
        if (T.rank_ >= T.K_) return true;
      }
    }
    // ---- build
    if constexpr (X::kResident) {
      __syncthreads();   // the list is this block's own work
      if (res_v == 0) {
        res_v = V;
        for (int32_t i = threadIdx.x; i < V; i += NT) W.comp[i] = i;
      }
      if (!list_here) {
#pragma unroll 4
        for (int64_t e = threadIdx.x; e < E; e += NT) {
          const int32_t u = L.src[e], d = L.dst[e];
          const float x = L.w[e];
          W.src[e] = u;
          W.dst[e] = d;
          W.w[e] = x;
        }
      }
      L = List{W.src, W.dst, W.w, 2.0f};
    }
#pragma unroll 1
    for (int32_t i = T.gt(); i < V; i += T.stride()) {
      W.k[i] = 0.0;
      W.loopw[i] = 0.0f;
      W.hasl[i] = 0;
    }
    if (lead) {
      W.ctl->flags = W.ctl->flags2 = W.ctl->check = W.ctl->loops = W.ctl->nlong = 0u;
      W.ctl->sums[0] = W.ctl->sums[1] = 0ull;
    }
    if (!T.sync()) return false;
    bool any_order = false;
    if (!at.symmetric) {
      check_list<X>(T, L, E, V);
      if (!T.sync()) return false;
      const uint32_t f = W.ctl->check;
      if (f & fBad) { at.bad = true; return true; }
      any_order = f != 0u || W.ctl->sums[0] != 0ull || W.ctl->sums[1] != 0ull;
      if (any_order && (X::kResident || !J.dbl)) { at.open = true; return true; }
      at.any_order = any_order;
    }
    if constexpr (!X::kResident) {
      if (threadIdx.x == 0) S.ngap = 0;
      __syncthreads();
    }
    // The list of rows M, of EM entries: the list itself, or its CSR.
    List M = L;
    int64_t EM = E;
    bool sparse = E < 2 * (int64_t)V;
    if constexpr (!X::kResident) {
      if (any_order) {
        EM = V <= (1 << 16) ? build_csr<X, uint32_t>(T, L, E, V) : build_csr<X, uint64_t>(T, L, E, V);
        if (EM < 0) return false;
        M = List{W.csrc, W.cdst, W.cw, 1.0f};
        sparse = EM < 2 * (int64_t)V;
        if (sparse) search_starts<X>(T, M.src, EM, V);
        uint32_t f = 0;
#pragma unroll 1
        for (int64_t e = T.gt(); e < EM; e += T.stride()) {
          const int32_t u = M.src[e], up = e > 0 ? M.src[e - 1] : -1;
          if (!sparse) {
            row_starts<X>(up + 1, u, (int32_t)e);
            if (e == EM - 1) row_starts<X>(u + 1, V, (int32_t)EM);
          }
          const float x = M.w[e];
          if (x != truncf(x)) f |= fNotInt;
        }
        if (f) atomicOr(&W.ctl->flags, f);
      }
    }
    if (!any_order) {
      if constexpr (!X::kResident) {
        if (sparse) search_starts<X>(T, L.src, E, V);
      }
      uint32_t f = 0, nl = 0;
#pragma unroll 1
      for (int64_t e0 = (int64_t)T.rank() * NT; e0 < E; e0 += T.stride()) {
        const int64_t e = e0 + threadIdx.x;
        if (e0 + (threadIdx.x & ~31) >= E) break;   // whole warps
        const bool in = e < E;
        const int32_t u = in ? L.src[e] : -1, d = in ? L.dst[e] : -2;
        const int32_t up = in && e > 0 ? L.src[e - 1] : -1;
        const float x = in ? L.w[e] : 0.0f;
        if (in) {
          if (X::kResident || !sparse) {
            row_starts<X>(up + 1, u, (int32_t)e);
            if (e == E - 1) row_starts<X>(u + 1, V, (int32_t)E);
          }
          if (x != truncf(x)) f |= fNotInt;
          if (u == d) { W.loopw[u] = x; W.hasl[u] = 1; ++nl; }
        }
        float g = x == 0.0f ? 1.0f : x;             // InitKernel.cu:165-170, both copies of the entry
        if (u == d) g *= 2.0f;
        bool run_last;
        const int depth = run_depth(u, run_last);
        double s = in ? __dadd_rn((double)g, (double)g) : 0.0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double t = __shfl_up_sync(0xffffffffu, s, o);
          if (o <= depth) s = __dadd_rn(s, t);
        }
        if (in && run_last) atomicAdd(&W.k[u], s);
      }
      f = __reduce_or_sync(0xffffffffu, f);
      nl = __reduce_add_sync(0xffffffffu, nl);
      if ((threadIdx.x & 31) == 0) {
        if (f) atomicOr(&W.ctl->flags, f);
        if (nl) atomicAdd(&W.ctl->loops, nl);
      }
    }
    if constexpr (!X::kResident) long_gaps<X>();
    group_partials<X>(   // NeighbourCompute.cu:46
        T, E, W.mpart, [&](int64_t e) { return L.w[e]; }, [&](int64_t, float x) { return (double)x; });
    if (!T.sync()) return false;
    const bool integral = !(W.ctl->flags & fNotInt);
    // of the next list: exact sums round alike in both directions
    at.symmetric = integral && !any_order;
    const int64_t nnz = EM - (int64_t)W.ctl->loops;
    const double m = finish_sum<X>(W.mpart, E);
    const double twom = __dmul_rn(2.0, m);
    {
      uint32_t f = 0;
      group_partials<X>(
          T, V, W.qpart, [&](int64_t i) { return Row{W.k[i], W.loopw[i], W.roff[i + 1] - W.roff[i]}; },
          [&](int64_t i, const Row& r) {
            const double x = (double)r.loopw;
            W.comm[i] = (int32_t)i;                 // InitKernel.cu:213-215
            W.next[i] = (int32_t)i;
            W.tot[i] = r.k;                         // InitKernel.cu:236
            W.in[i] = x;                            // InitKernel.cu:242
            W.size[i] = 1;                          // OneLevelKernel.cu:87
            delta_clear(W.delta[i]);
            W.cand[i] = -1;
            W.kfrac[i] = m > 0.0 ? __ddiv_rn(r.k, twom) : 0.0;   // OneLevelKernel.cu:307
            W.minidx[i] = kNone;
            if constexpr (!X::kResident) {
              if (r.len > Tile<NT>::kF64) {
                f |= fLong;
                W.longs[atomicAdd(&W.ctl->nlong, 1u)] = (int32_t)i;
              }
            }
            if (!(r.k < 1073741824.0)) f |= fNotInt;
            return q_term(x, r.k, m, twom);
          });
      if (f) atomicOr(&W.ctl->flags2, f);
    }
    if (!T.sync()) return false;
    const uint32_t f2 = W.ctl->flags2;
    const bool packed = integral && !(f2 & fNotInt);
    const bool longs = !X::kResident && (f2 & fLong);
    const double q0 = finish_sum<X>(W.qpart, V);
    const double lower = level == 0 ? q0 : at.mod;   // LouvainCPP.cpp:356,446
    find_rows<X>(T, V, EM);
    const int32_t v0 = S.row0, v1 = S.row1;
    const long long t1 = clock64();
    // ---- passes
    double q_prev = q0, floor_q = -1.0;         // curMod = -1 (OneLevelKernel.cu:528)
    int pass = 1, st = LVG_OK;
    float pass_ticks[2] = {0.0f, 0.0f};
#pragma unroll 1
    for (;; ++pass) {
      const long long p0 = clock64();
      // the pass's test uses the Q of the state before it, so it is known here
      // (OneLevelKernel.cu:889-896): the pass that ends the level keeps its
      // decisions but not their totals
      const bool stop = __dsub_rn(q_prev, floor_q) < cfg.pass_min;
      const bool capped = cfg.max_passes >= 0 && pass >= cfg.max_passes;
      if (pass == 1) {
        if constexpr (!X::kResident) {
          if (longs) hub_clear<X>(T);
        }
        moves_first<X>(M, v0, v1, stop || capped);
      } else if (packed) {
        moves_hash<X, true>(M, v0, v1, stop || capped);
      } else {
        moves_hash<X, false>(M, v0, v1, stop || capped);
      }
      if constexpr (!X::kResident) {
        if (longs && pass > 1) {
          if (packed) hub_insert<X, true>(T, M, EM);
          else hub_insert<X, false>(T, M, EM);
        }
      }
      if (!T.sync()) return false;
      if constexpr (!X::kResident) {
        if (longs && pass > 1) {
          if (packed) hub_pick<X, true>(T, stop || capped);
          else hub_pick<X, false>(T, stop || capped);
          if (!T.sync()) return false;
        }
      }
      if (pass <= 2) pass_ticks[pass - 1] = (float)(clock64() - p0);
      else if (lead && J.pass_ticks) J.pass_ticks[pass - 1] = (float)(clock64() - p0);
      if (stop || capped) {
        st = stop ? LVG_OK : LVG_ERR_NOT_CONVERGED;
        break;
      }
      commit<X, false>(T, V, m);
      if (!T.sync()) return false;
      const double q = finish_sum<X>(W.qpart, V);
      floor_q = q_prev < lower ? lower : q_prev;
      q_prev = q;
      if (pass >= kSmallPassCap) { at.open = true; return true; }
    }
#pragma unroll 1
    for (int32_t i = T.gt(); i < V; i += T.stride()) {      // isolated merge (OneLevelKernel.cu:138-171)
      const int32_t c = W.cand[i];
      if (c >= 0) {
        W.next[i] = c;
        move_deltas<false>(W.delta, W.comm[i], c, W.k[i], __dadd_rn(0.0, (double)W.loopw[i]));
      }
    }
    if (!T.sync()) return false;
    commit<X, true>(T, V, m);
    if (!T.sync()) return false;
    const double ql = finish_sum<X>(W.qpart, V);
    const long long t2 = clock64();
    // ---- renumber by smallest member (RenumberKernel.cu:121-133)
    const int32_t i0 = (int32_t)((int64_t)V * T.rank() / T.K()), i1 = (int32_t)((int64_t)V * (T.rank() + 1) / T.K());
    uint32_t run = 0, C = 0;
    if (T.K() > 1) {
      uint32_t heads = 0;
#pragma unroll 1
      for (int32_t b0 = i0; b0 < i1; b0 += NT) {
        const int32_t i = b0 + threadIdx.x;
        heads += __syncthreads_count(i < i1 && W.minidx[W.comm[i < i1 ? i : i0]] == i);
      }
      if (threadIdx.x == 0) W.ctl->count[0][T.rank()] = heads;
      if (!T.sync()) return false;
#pragma unroll 4
      for (int r = 0; r < T.K(); ++r) {
        const uint32_t c = W.ctl->count[0][r];
        if (r < T.rank()) run += c;
        C += c;
      }
    }
    {
      uint32_t at_run = run;
#pragma unroll 1
      for (int32_t b0 = i0; b0 < i1; b0 += NT) {
        const int32_t i = b0 + threadIdx.x;
        const int32_t c = i < i1 ? W.comm[i] : 0;
        const bool h = i < i1 && W.minidx[c] == i;
        uint32_t all;
        const uint32_t ex = block_excl<X>(h ? 1u : 0u, &all);
        if (h) W.newid[c] = (int32_t)(at_run + ex);
        at_run += all;
      }
      if (T.K() == 1) C = at_run;
    }
    if (!T.sync()) return false;
    if (J.parts) {
      int32_t* part = J.parts + (J.parts_cap - at.part_off - 2 * (int64_t)V);
#pragma unroll 1
      for (int32_t i = T.gt(); i < V; i += T.stride()) {
        const int32_t c = W.comm[i];
        part[i] = W.newid[c];
        part[V + i] = c;
      }
    }
    if constexpr (X::kResident) {
      for (int32_t i = threadIdx.x; i < res_v; i += NT) W.comp[i] = W.newid[W.comm[W.comp[i]]];
    } else {
#pragma unroll 2
      for (int32_t i = T.gt(); i < J.V; i += T.stride())     // partitionAtLevel (LouvainCPP.cpp:82-106)
        J.comp[i] = W.newid[W.comm[at.nlev == 0 ? i : J.comp[i]]];
    }
    const long long t3 = clock64();
    // ---- level break (LouvainCPP.cpp:466)
    bool last = false;
    if (st != LVG_OK) { at.status = st; last = true; }
    else if (level > 0 && (ql - at.mod) < cfg.level_min) last = true;
    else if (cfg.max_levels >= 0 && level + 1 >= cfg.max_levels) { at.status = LVG_ERR_NOT_CONVERGED; last = true; }
    if (last && J.state) keep_state<X>(T, V, J.state);
    at.mod = ql;
    int64_t E1 = 0;
    int32_t *ns = nullptr, *nd = nullptr;
    float* nw = nullptr;
    if (!last) {
      list_of(J.lists, J.E, at.nlev & 1, &ns, &nd, &nw);
      if (X::kResident || C <= (1u << 16)) E1 = coarsen<X, uint32_t>(T, L, E, (int32_t)C, packed, ns, nd, nw);
      else E1 = coarsen<X, uint64_t>(T, L, E, (int32_t)C, packed, ns, nd, nw);
      if (E1 < 0) return false;
    }
    if (lead && J.lv) {
      SmallLevel& R = J.lv[at.nlev];
      R.V = V;
      R.C = (int32_t)C;
      R.passes = pass;
      R.E = E;
      R.nnz = nnz;
      R.q_start = q0;
      R.q_level = ql;
      R.ticks[0] = (float)(t1 - t0);
      R.ticks[1] = (float)(t2 - t1);
      R.ticks[2] = (float)(t3 - t2);
      R.ticks[3] = last ? 0.0f : (float)(clock64() - t3);
      R.pass_ticks[0] = pass_ticks[0];
      R.pass_ticks[1] = pass_ticks[1];
      R.part_off = J.parts_cap - at.part_off - 2 * (int64_t)V;
    }
    at.part_off += 2 * (int64_t)V;
    at.ncomms = (int32_t)C;
    ++at.nlev;
    if (last) return true;
    at.buf = (at.nlev - 1) & 1;
    L = List{ns, nd, nw, 2.0f};
    list_here = cells_fit<X>((int32_t)C);
    at.V = (int32_t)C;
    at.E = E1;
  }
}

template <typename X>
__device__ __forceinline__ void load_job(const SmallJob* job) {
  static_assert(sizeof(SmallJob) % 4 == 0 && sizeof(SmallJob) / 4 <= X::NT, "a word a thread");
  if (threadIdx.x < sizeof(SmallJob) / 4)
    reinterpret_cast<uint32_t*>(&X::S().J)[threadIdx.x] = reinterpret_cast<const uint32_t*>(job)[threadIdx.x];
  __syncthreads();
}

__device__ __forceinline__ void store_between(Between& B, const At& at) {
  B.nlev = at.nlev;
  B.buf = at.buf;
  B.symmetric = (at.symmetric ? 1 : 0) | (at.any_order ? 2 : 0);
  B.V = at.V;
  B.ncomms = at.ncomms;
  B.open = at.open ? 1 : 0;
  B.bad = at.bad ? 1 : 0;
  B.status = at.status;
  B.E = at.E;
  B.part_off = at.part_off;
  B.mod = at.mod;
}

__device__ __forceinline__ void load_between(const Between& B, At& at) {
  at.V = B.V;
  at.E = B.E;
  at.ncomms = B.ncomms;
  at.buf = B.buf;
  at.nlev = B.nlev;
  at.symmetric = (B.symmetric & 1) != 0;
  at.any_order = (B.symmetric & 2) != 0;
  at.mod = B.mod;
  at.part_off = B.part_off;
}

// First launch (and the second, a cluster's, behind a grid's): the levels
// until one fits a block's shared memory.
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) small_kernel(const SmallJob* jobs, int K, int mode, int resume,
                                                               SmallCfg cfg) {
  using X = Multi<NT>;
  if (mode == kModeGrid && (int)blockIdx.x == cfg.hold) return;
  load_job<X>(jobs + blockIdx.x / K);
  const SmallJob& J = X::S().J;
  if (threadIdx.x == 0) {
    carve(J.work, J.V, J.E, J.dbl != 0, J.blocks, X::W());
    X::S().goal = 0ull;
    X::S().wait_ns = (unsigned long long)cfg.wait_ns;
  }
  __syncthreads();
  Team<X> T{K, (int)(blockIdx.x % K), mode};
  const unsigned long long ns0 = now_ns();
  const long long c0 = clock64();
  At at;
  at.V = J.V;
  at.E = J.E;
  at.symmetric = J.check == 0;
  at.any_order = J.dbl != 0;
  at.mod = J.mod;
  Between& B = *X::W().bt;
  if (resume) {   // from where the grid stopped
    if (B.phase != kPhaseMid) return;
    load_between(B, at);
    if (!T.sync()) return;   // before the first block writes it again
  }
  if (!run_levels<X>(T, cfg, at)) return;
  if (T.lead()) {
    store_between(B, at);
    const long long ticks = clock64() - c0;
    B.ms_per_tick = ticks > 0 ? 1e-6 * (double)(now_ns() - ns0) / (double)ticks : 0.0;
    B.comp = kCompDone;
    B.phase = at.mid ? kPhaseMid : at.tail ? kPhaseTail : kPhaseEnd;
  }
}

// Second launch, a block per job: the levels that fit its shared memory, and
// the sums of the modularity cleared.
__global__ void __launch_bounds__(kResThreads, 1) small_tail_kernel(const SmallJob* jobs, SmallCfg cfg) {
  using X = Tail;
  load_job<X>(jobs + blockIdx.x);
  const SmallJob& J = X::S().J;
  Work g;
  carve(J.work, J.V, J.E, J.dbl != 0, J.blocks, g);
  Between& B = *g.bt;
  const int32_t phase = B.phase;
  int32_t ncomms = B.ncomms;
  if (phase == kPhaseTail) {
    if (threadIdx.x == 0) {
      Resident& W = X::W();
      W.key[0] = g.key[0];
      W.key[1] = g.key[1];
      W.val[0] = g.val[0];
      W.val[1] = g.val[1];
      W.wsum = g.wsum;
      W.ghist = g.ghist;
    }
    At at;
    load_between(B, at);
    const bool first = at.nlev == 0;
    const int32_t nlev0 = at.nlev, v0 = at.V;
    __syncthreads();
    Team<X> T{1, 0, kModeCluster};
    run_levels<X>(T, cfg, at);
    ncomms = at.ncomms;
    const bool any = at.nlev > nlev0;
    if (any)
      for (int32_t i = threadIdx.x; i < v0; i += kResThreads) g.rc[i] = X::W().comp[i];
    if (threadIdx.x == 0) {
      store_between(B, at);
      B.comp = !any ? kCompDone : (first ? kCompTailAll : kCompTail);
      B.phase = kPhaseEnd;
    }
  }
  if (J.want_q)
    for (int32_t i = threadIdx.x; i < ncomms; i += kResThreads) g.tot[i] = g.in[i] = 0.0;
}

__device__ __forceinline__ int32_t final_comm(const SmallJob& J, const Work& g, int32_t how, int32_t i) {
  return how == kCompDone ? J.comp[i] : g.rc[how == kCompTailAll ? i : J.comp[i]];
}

__device__ __forceinline__ bool wants_q(const SmallJob& J, const Between& B) {
  return J.want_q && B.phase == kPhaseEnd && !B.open && !B.bad;
}

constexpr int kQThreads = 512;

// Third launch (K blocks a job): community strengths and internal weights of
// the final communities over the job's list, as nm_accum_kernel<true>: the list
// is symmetric, so each entry adds 2w to its source's community.
__global__ void __launch_bounds__(kQThreads) small_sum_kernel(const SmallJob* jobs, int K) {
  const SmallJob& J = jobs[blockIdx.x / K];
  Work g;
  carve(J.work, J.V, J.E, J.dbl != 0, J.blocks, g);
  const Between& B = *g.bt;
  if (!wants_q(J, B)) return;
  const int32_t how = B.comp;
  const int64_t stride = (int64_t)K * kQThreads;
#pragma unroll 2
  for (int64_t e0 = (int64_t)(blockIdx.x % K) * kQThreads; e0 < J.E; e0 += stride) {
    const int64_t e = e0 + threadIdx.x;
    const bool in = e < J.E;
    const int32_t u = in ? J.src[e] : -1;
    const double x = in ? 2.0 * (double)J.w[e] : 0.0;
    const int32_t a = in ? final_comm(J, g, how, u) : -1, b = in ? final_comm(J, g, how, J.dst[e]) : -1;
    bool run_last;
    const int depth = run_depth(u, run_last);
    double kin = x, ain = a == b ? x : 0.0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t1 = __shfl_up_sync(0xffffffffu, kin, o), t2 = __shfl_up_sync(0xffffffffu, ain, o);
      if (o <= depth) {
        kin = __dadd_rn(kin, t1);
        ain = __dadd_rn(ain, t2);
      }
    }
    if (in && run_last) {
      atomicAdd(&g.tot[a], kin);
      if (ain != 0.0) atomicAdd(&g.in[a], ain);
    }
  }
}

struct QSpace {
  static constexpr int NT = kQThreads;
  static constexpr bool kResident = true;
  struct Smem {
    union {
      double stage[kGroup];
    } u;
    double ws[8];
    double bcast;
  };
  static __device__ __forceinline__ Smem& S() { return *reinterpret_cast<Smem*>(smem_raw); }
};

// Fourth launch (K blocks a job): the composition of the tail's levels; the
// job's first block takes the modularity and writes the result.
__global__ void __launch_bounds__(kQThreads) small_end_kernel(const SmallJob* jobs, int K) {
  const SmallJob& J = jobs[blockIdx.x / K];
  Work g;
  carve(J.work, J.V, J.E, J.dbl != 0, J.blocks, g);
  const Between& B = *g.bt;
  if (B.phase != kPhaseEnd) return;   // a barrier's wait ran out: no result
  const int32_t how = B.comp;
  if (how != kCompDone)
    for (int64_t i = (int64_t)(blockIdx.x % K) * kQThreads + threadIdx.x; i < J.V; i += (int64_t)K * kQThreads)
      J.comp[i] = final_comm(J, g, how, (int32_t)i);
  if (blockIdx.x % K != 0) return;
  double q = 0.0;
  if (wants_q(J, B)) {
    const Team<QSpace> T{1, 0, kModeCluster};
    const int64_t C = B.ncomms;
    group_partials<QSpace>(
        T, C, g.mpart, [&](int64_t c) { return g.tot[c]; }, [&](int64_t, double x) { return x; });
    __syncthreads();
    const double tw = finish_sum<QSpace>(g.mpart, C);
    group_partials<QSpace>(
        T, C, g.qpart, [&](int64_t c) { return make_double2(g.tot[c], g.in[c]); },
        [&](int64_t, const double2& x) {
          const double f = __ddiv_rn(x.x, tw);
          return tw > 0.0 ? __dsub_rn(__ddiv_rn(x.y, tw), __dmul_rn(f, f)) : 0.0;
        });
    __syncthreads();
    q = finish_sum<QSpace>(g.qpart, C);
  }
  if (threadIdx.x == 0) {
    SmallResult& O = *J.res;
    O.n_levels = B.nlev;
    O.n_comms = B.ncomms;
    O.open = B.open;
    O.status = B.status;
    O.bad = B.bad;
    O.V = B.V;
    O.buf = B.buf;
    O.E = B.E;
    O.ms_per_tick = B.ms_per_tick;
    O.mod = B.mod;
    O.q_final = q;
    O.finished = 1;
  }
}

void set_attributes() {
  constexpr int kDevs = 64;
  static std::mutex mu;
  static bool done[kDevs] = {};
  int dev = 0;
  LVG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (dev >= 0 && dev < kDevs && done[dev]) return;
  constexpr auto kSmem = cudaFuncAttributeMaxDynamicSharedMemorySize;
  LVG_CUDA(cudaFuncSetAttribute(small_kernel<512>, kSmem, (int)sizeof(Multi<512>::Smem)));
  LVG_CUDA(cudaFuncSetAttribute(small_kernel<1024>, kSmem, (int)sizeof(Multi<1024>::Smem)));
  LVG_CUDA(cudaFuncSetAttribute(small_kernel<1024>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  LVG_CUDA(cudaFuncSetAttribute(small_tail_kernel, kSmem, (int)sizeof(Tail::Smem)));
  if (dev >= 0 && dev < kDevs) done[dev] = true;
}

// Test hook (lvg_debug_small_launch): the error every launch of the levels meets.
std::atomic<int32_t> g_launch_error{0};
// Test hook (lvg_debug_small_hold): a block that stays away from the grid's
// barriers, and their limit.
std::atomic<int32_t> g_hold{-1};
std::atomic<int64_t> g_wait_ns{SmallCfg().wait_ns};

// False: such a launch is refused here (a cluster or a grid that must be on
// the chip together, on a stream that may use a part of the chip).
template <int NT>
bool launch_levels(const SmallJob* jobs, int n, int K, int mode, int resume, const SmallCfg& cfg, cudaStream_t s) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)(n * K));
  lc.blockDim = dim3(NT);
  lc.dynamicSmemBytes = sizeof(typename Multi<NT>::Smem);
  lc.stream = s;
  cudaLaunchAttribute at[1];
  if (mode == kModeGrid) {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  } else {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)K;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
  }
  lc.attrs = at;
  lc.numAttrs = mode == kModeGrid || K > 1 ? 1 : 0;
  cudaError_t e = (cudaError_t)g_launch_error.load();
  if (e == cudaSuccess) e = cudaLaunchKernelEx(&lc, small_kernel<NT>, jobs, K, mode, resume, cfg);
  switch (e) {
    case cudaErrorCooperativeLaunchTooLarge:
    case cudaErrorInvalidClusterSize:
    case cudaErrorLaunchOutOfResources:
    case cudaErrorInvalidConfiguration:
    case cudaErrorNotSupported:
      cudaGetLastError();
      return false;
    default:
      LVG_CUDA(e);
  }
  count_launch();
  return true;
}

// The launches behind the levels: the tail, and the results by K blocks a job.
void launch_rest(const SmallJob* jobs, int n, int K, const SmallCfg& cfg, cudaStream_t s) {
  small_tail_kernel<<<(unsigned)n, kResThreads, sizeof(Tail::Smem), s>>>(jobs, cfg);
  LVG_LAUNCH();
  small_sum_kernel<<<(unsigned)(n * K), kQThreads, 0, s>>>(jobs, K);
  LVG_LAUNCH();
  small_end_kernel<<<(unsigned)(n * K), kQThreads, sizeof(QSpace::Smem), s>>>(jobs, K);
  LVG_LAUNCH();
}

}  // namespace

size_t small_list_bytes(int64_t E) { return 6 * up256(4 * (size_t)E); }

size_t small_work_bytes(int32_t V, int64_t E, bool dbl, int blocks) {
  Work W;
  return carve(nullptr, V, E, dbl, blocks, W);
}

void small_list(char* lists, int64_t E, int buf, int32_t** src, int32_t** dst, float** w) {
  list_of(lists, E, buf, src, dst, w);
}

bool small_fits(int64_t V, int64_t E, int64_t max_entries) {
  return V > 0 && V <= kSmallMaxV && E > 0 && E <= max_entries;
}

bool small_run(const SmallJob* d_jobs, int n, int K, const SmallCfg& cfg, cudaStream_t s) {
  if (n <= 0) return true;
  set_attributes();
  if (!(K >= 8 ? launch_levels<1024>(d_jobs, n, K, kModeCluster, 0, cfg, s)
               : launch_levels<512>(d_jobs, n, K, kModeCluster, 0, cfg, s)))
    return false;
  launch_rest(d_jobs, n, K, cfg, s);
  return true;
}

int small_grid_blocks() {
  constexpr int kDevs = 64;
  static std::mutex mu;
  static int blocks[kDevs] = {};
  set_attributes();
  int dev = 0;
  LVG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (dev >= 0 && dev < kDevs && blocks[dev] > 0) return blocks[dev];
  int sms = 0, per = 0;
  LVG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  LVG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, small_kernel<1024>, 1024, sizeof(Multi<1024>::Smem)));
  const int n = std::min(sms * std::min(per, 1), kSmallMaxBlocks);
  if (dev >= 0 && dev < kDevs) blocks[dev] = n;
  return n;
}

bool small_run_grid(const SmallJob* d_job, void* work, int K, const SmallCfg& given, cudaStream_t s) {
  SmallCfg cfg = given;
  cfg.hold = g_hold.load();
  cfg.wait_ns = g_wait_ns.load();
  // the barrier's words, and the phase, should a wait run out
  LVG_CUDA(cudaMemsetAsync(work, 0, up256(sizeof(Ctl)) + up256(sizeof(Between)), s));
  set_attributes();
  if (!launch_levels<1024>(d_job, 1, K, kModeGrid, 0, cfg, s)) return false;
  // (refused, it leaves levels that the grid did not finish undone: no result)
  launch_levels<1024>(d_job, 1, kSmallClusterBlocks, kModeCluster, 1, cfg, s);
  launch_rest(d_job, 1, K, cfg, s);
  return true;
}

}  // namespace lvg

extern "C" lvg_status lvg_debug_small_launch(int32_t error) {
  lvg::g_launch_error.store(error);
  return LVG_OK;
}

extern "C" lvg_status lvg_debug_small_hold(int32_t block, int64_t wait_ns) {
  if (wait_ns < 0) return LVG_ERR_INVALID_ARG;
  lvg::g_hold.store(block);
  lvg::g_wait_ns.store(wait_ns > 0 ? wait_ns : lvg::SmallCfg().wait_ns);
  return LVG_OK;
}
