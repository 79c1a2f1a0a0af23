// Device-wide primitives: scans, fixed-tree sums, stable LSD radix sort.
//
// Radix sort (replaces thrust::sort_by_key on zip keys, NeighbourCompute.cu:82,
// InducedGraphKernel.cu:91): stable LSD, 8-bit digits.  One upfront pass over
// the keys counts every digit position; then one kernel per digit: a
// 4096-key tile (taken in launch order from a counter) ranks its keys stably
// in shared memory (the lanes of a digit meet in a shared word), learns the counts of
// its digits in all earlier tiles by decoupled look-back (bounded spin, error
// flag), and writes its keys out digit run by digit run.
#include <algorithm>
#include <atomic>
#include <mutex>

#include "prims.cuh"

namespace lvg {
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T* total) {
  static_assert(kScanThreads == 256, "block scan assumes 256 threads");
  return block_exclusive_scan256<T>(v, total);
}

struct AddOp {
  template <typename T> static __device__ __forceinline__ T of(T a, T b) { return a + b; }
};
struct MaxOp {   // of values >= 0
  template <typename T> static __device__ __forceinline__ T of(T a, T b) { return a > b ? a : b; }
};

// Exclusive scan of one value per thread over the block, and its total.
template <typename Op, typename T>
__device__ __forceinline__ T block_exclusive_op(T v, T* total) {
  __shared__ T wsum[8];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T u = __shfl_up_sync(full, inc, o);
    if (lane >= o) inc = Op::of(u, inc);
  }
  if (lane == 31) wsum[w] = inc;
  __syncthreads();
  T base = T(0), tot = T(0);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (k < w) base = Op::of(base, wsum[k]);
    tot = Op::of(tot, wsum[k]);
  }
  *total = tot;
  __syncthreads();
  T ex = __shfl_up_sync(full, inc, 1);
  if (lane == 0) ex = T(0);
  return Op::of(base, ex);
}

template <typename Op, typename T>
__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const T* in, int64_t n, T* bsum) {
  int64_t base = (int64_t)blockIdx.x * kScanTile + threadIdx.x;
  T s = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j)   // any order: the block's total alone
    if (base + j * kScanThreads < n) s = Op::of(s, in[base + j * kScanThreads]);
  T tot;
  block_exclusive_op<Op, T>(s, &tot);
  if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

template <typename Op, typename T>
__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(const T* in, T* out, int64_t n,
                                                                  const T* bscan) {
  int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  T v[kScanItems];
  T s = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    v[j] = base + j < n ? in[base + j] : T(0);
    s = Op::of(s, v[j]);
  }
  T tot;
  T pre = block_exclusive_op<Op, T>(s, &tot);
  const T before = bscan ? bscan[blockIdx.x] : T(0);
  T off = Op::of(before, pre);
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    if (base + j < n) out[base + j] = off;
    off = Op::of(off, v[j]);
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = Op::of(before, tot);
}

template <typename Op, typename T>
void scan_impl(const T* in, T* out, int64_t n, Arena& a, cudaStream_t s) {
  if (n <= 0) {
    LVG_CUDA(cudaMemsetAsync(out, 0, sizeof(T), s));
    return;
  }
  HiScope hs(a);
  int64_t nb = (n + kScanTile - 1) / kScanTile;
  T* bscan = nullptr;
  if (nb > 1) {
    T* bsum = a.hi_n<T>(nb + 1);
    scan_reduce_kernel<Op, T><<<(unsigned)nb, kScanThreads, 0, s>>>(in, n, bsum);
    LVG_LAUNCH();
    scan_impl<Op, T>(bsum, bsum, nb, a, s);
    bscan = bsum;
  }
  scan_apply_kernel<Op, T><<<(unsigned)nb, kScanThreads, 0, s>>>(in, out, n, bscan);
  LVG_LAUNCH();
}

// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kRedThreads) tree_group_kernel(const T* x, int64_t n, double* out) {
  __shared__ double ws[8];
  int64_t b = blockIdx.x;
  int64_t len = n - b * kGroup;
  if (len > kGroup) len = kGroup;
  double r = group_sum_block<T>(x + b * kGroup, len, ws);
  if (threadIdx.x == 0) out[b] = r;
}

void finish_impl(const double* p, int64_t n, double* d_out, Arena& a, cudaStream_t s) {
  HiScope hs(a);
  while (n > 1) {
    int64_t nb = (n + kGroup - 1) / kGroup;
    double* q = nb == 1 ? d_out : a.hi_n<double>(nb);
    tree_group_kernel<double><<<(unsigned)nb, kRedThreads, 0, s>>>(p, n, q);
    LVG_LAUNCH();
    p = q;
    n = nb;
  }
}

// ---------------------------------------------------------------------------
constexpr int kRsThreads = 256;
constexpr int kRsItems = 16;
constexpr int kRsTile = kRsThreads * kRsItems;  // 4096 keys
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRadix = 256;

// One pass over the keys gives the global histogram of every digit position.
constexpr int kRsMaxPasses = 8;

__global__ void __launch_bounds__(kRsThreads) rs_upfront_kernel(const uint64_t* keys, int64_t n, int lo, int bits,
                                                                int npass, uint32_t* ghist) {
  __shared__ uint32_t h[kRsMaxPasses][kRadix];
  for (int i = threadIdx.x; i < kRsMaxPasses * kRadix; i += kRsThreads) (&h[0][0])[i] = 0;
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)kRsThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kRsThreads) {
    const uint64_t k = bits < 64 ? (keys[i] >> lo) & ((1ull << bits) - 1ull) : keys[i] >> lo;
    for (int p = 0; p < npass; ++p) atomicAdd(&h[p][(unsigned)(k >> (8 * p)) & (kRadix - 1)], 1u);
  }
  __syncthreads();
  for (int p = 0; p < npass; ++p) {
    const uint32_t c = h[p][threadIdx.x];
    if (c) atomicAdd(&ghist[p * kRadix + threadIdx.x], c);
  }
}

// Exclusive scan of each pass's global histogram (one block, thread = digit).
__global__ void __launch_bounds__(kRsThreads) rs_gscan_kernel(uint32_t* ghist, int npass) {
  for (int p = 0; p < npass; ++p) {
    uint32_t tot;
    const uint32_t v = ghist[p * kRadix + threadIdx.x];
    const uint32_t x = block_exclusive_scan<uint32_t>(v, &tot);
    __syncthreads();
    ghist[p * kRadix + threadIdx.x] = x;
    __syncthreads();
  }
}

template <bool VALS>
struct RsSmem {
  uint64_t key[kRsTile];
  float val[VALS ? kRsTile : 1];
  uint32_t wc[kRsWarps][kRadix];     // keys of the digit so far, then its first staged position
  uint32_t peers[kRsWarps][kRadix];  // lanes of the round's keys with the digit
  uint32_t gbase[kRadix];
  uint32_t tile;
};

// Look-back words, one per (tile, digit): code in bits 56..63 (2p+1: this
// tile's count, 2p+2: count of every tile up to this one, for pass p; codes of
// earlier passes read as "not yet"), count in bits 0..31.
constexpr int kRsWindow = 8;
constexpr int kRsSpinLimit = 1 << 22;
// Test hook (lvg_debug_radix_hold): a smaller spin limit and one tile that
// never publishes, so that the bounded wait of its successors runs out.
std::atomic<int> g_rs_spin_limit{kRsSpinLimit};
std::atomic<int64_t> g_rs_hold_tile{-1};

__device__ __forceinline__ void rs_publish(unsigned long long* w, unsigned code, uint32_t count) {
  atomicExch(w, ((unsigned long long)code << 56) | count);
}

// One LSD pass: a tile (taken in launch order from a counter) ranks its keys
// by digit in shared memory, learns the keys of its digits in all earlier
// tiles by decoupled look-back, and writes its keys out digit run by digit
// run.  Stable: ranks follow key order inside a tile and tiles in order.
//
// Bound by shared memory (the coarsening's passes on R-MAT scale 20, 31.4 M
// keys: the L1 data stage 60 to 69 % busy, DRAM 23 to 25 %).  So nothing is
// looked up twice: ranks and staged positions are kept in 16 bits, a digit's
// lanes meet in one word (an atomic or, where a match instruction was the
// slower), and what can be packed into the key's free bits comes without
// values (lists of whole weights, induce.cu).  Three tiles fit an SM (two
// before); the look-back reads kRsWindow tiles at a time.
// 134 M random keys, three passes: 4.81 -> 3.84 ms, 2.96 ms without values.
template <bool VALS>
__global__ void __launch_bounds__(kRsThreads, 3) rs_onesweep_kernel(
    const uint64_t* kin, const float* vin, uint64_t* kout, float* vout, int64_t n, int shift, uint32_t dmask,
    int pass, const uint32_t* gstart, unsigned long long* look, uint32_t* counter, uint32_t* err, int spin_limit,
    int64_t hold) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RsSmem<VALS>& S = *reinterpret_cast<RsSmem<VALS>*>(smem_raw);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) S.tile = atomicAdd(counter, 1u);
  for (int i = threadIdx.x; i < kRsWarps * kRadix; i += kRsThreads) (&S.wc[0][0])[i] = (&S.peers[0][0])[i] = 0;
  __syncthreads();
  const int64_t tile = S.tile;
  const int64_t tile0 = tile * kRsTile;
  const int tn = (int)min((int64_t)kRsTile, n - tile0);
  const int base = w * (32 * kRsItems) + lane;   // the lane's first key in the tile; its others 32 apart
  const uint64_t* kt = kin + tile0;
  uint64_t k[kRsItems];
  uint32_t pos2[kRsItems / 2];   // rank in the warp, then staged position, two to a word
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int j = 0; j < kRsItems; ++j) k[j] = base + j * 32 < tn ? kt[base + j * 32] : 0ull;
  auto digit = [&](uint64_t key) { return (unsigned)(key >> shift) & dmask; };
  // stable ranks inside the tile: the lanes holding a digit meet in its word
  // of shared memory
#pragma unroll
  for (int j = 0; j < kRsItems; ++j) {
    const bool in = base + j * 32 < tn;
    const unsigned dd = digit(k[j]);
    if (in) atomicOr(&S.peers[w][dd], 1u << lane);
    __syncwarp();
    const unsigned peers = in ? S.peers[w][dd] : 0u;
    const uint32_t before = S.wc[w][dd];
    const uint32_t r = before + __popc(peers & lt);
    pos2[j / 2] = (j & 1) ? pos2[j / 2] | (r << 16) : r;
    __syncwarp();
    if (in && (peers & lt) == 0) {
      S.wc[w][dd] = before + __popc(peers);
      S.peers[w][dd] = 0u;
    }
    __syncwarp();
  }
  __syncthreads();
  // thread = digit: the tile's count, published; the first staged position of
  // every warp's keys
  const int d = threadIdx.x;
  uint32_t cnt = 0;
#pragma unroll
  for (int ww = 0; ww < kRsWarps; ++ww) cnt += S.wc[ww][d];
  const unsigned agg = 2u * (unsigned)pass + 1u, inc = agg + 1u;
  unsigned long long* mine = look + tile * kRadix + d;
  const bool publish = tile != hold;   // hold: a test makes this tile's successors wait out their limit
  if (publish) rs_publish(mine, tile == 0 ? inc : agg, cnt);
  uint32_t tot;
  const uint32_t start = block_exclusive_scan<uint32_t>(cnt, &tot);
  uint32_t run = start;
#pragma unroll
  for (int ww = 0; ww < kRsWarps; ++ww) {
    const uint32_t t = S.wc[ww][d];
    S.wc[ww][d] = run;
    run += t;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRsItems; ++j)
    if (base + j * 32 < tn) {
      const uint32_t p = S.wc[w][digit(k[j])] + ((pos2[j / 2] >> (16 * (j & 1))) & 0xffffu);
      S.key[p] = k[j];
      if (VALS) pos2[j / 2] = (j & 1) ? (pos2[j / 2] & 0xffffu) | (p << 16) : (pos2[j / 2] & 0xffff0000u) | p;
    }
  if (VALS) {
    float v[kRsItems];
#pragma unroll
    for (int j = 0; j < kRsItems; ++j) v[j] = base + j * 32 < tn ? vin[tile0 + base + j * 32] : 0.0f;
#pragma unroll
    for (int j = 0; j < kRsItems; ++j)
      if (base + j * 32 < tn) S.val[(pos2[j / 2] >> (16 * (j & 1))) & 0xffffu] = v[j];
  }
  // keys of the digit in all earlier tiles
  uint32_t excl = 0;
  if (tile > 0) {
    int64_t j = tile - 1;
    int spins = 0;
    bool found = false;
    while (j >= 0 && !found) {
      unsigned long long x[kRsWindow];
#pragma unroll
      for (int q = 0; q < kRsWindow; ++q)
        x[q] = j - q >= 0 ? *reinterpret_cast<volatile unsigned long long*>(look + (j - q) * kRadix + d) : 0ull;
      bool ready = true;   // every tile of the window before this one
#pragma unroll
      for (int q = 0; q < kRsWindow; ++q) {
        const unsigned code = (unsigned)(x[q] >> 56);
        if (ready && !found && j >= 0) {
          if (code == inc || code == agg) {
            excl += (uint32_t)x[q];
            found = code == inc;
            --j;
          } else {
            ready = false;
          }
        }
      }
      if (!ready && ++spins > spin_limit) { atomicOr(err, 1u); break; }   // bounded wait: report, never hang
    }
    if (publish) rs_publish(mine, inc, excl + cnt);
  }
  S.gbase[d] = gstart[d] + excl - start;   // (mod 2^32) output position of the tile's staged position 0
  __syncthreads();
#pragma unroll 4
  for (int p = threadIdx.x; p < tn; p += kRsThreads) {
    const uint64_t kk = S.key[p];
    const uint32_t o = S.gbase[digit(kk)] + (uint32_t)p;
    kout[o] = kk;
    if (VALS) vout[o] = S.val[p];
  }
}

}  // namespace

void scan_u32(const uint32_t* in, uint32_t* out, int64_t n, Arena& a, cudaStream_t s) {
  scan_impl<AddOp, uint32_t>(in, out, n, a, s);
}
void scan_i64(const int64_t* in, int64_t* out, int64_t n, Arena& a, cudaStream_t s) {
  scan_impl<AddOp, int64_t>(in, out, n, a, s);
}
void scan_max_i64(const int64_t* in, int64_t* out, int64_t n, Arena& a, cudaStream_t s) {
  scan_impl<MaxOp, int64_t>(in, out, n, a, s);
}

void tree_sum_f64(const double* x, int64_t n, double* d_out, Arena& a, cudaStream_t s) {
  if (n <= 0) { LVG_CUDA(cudaMemsetAsync(d_out, 0, sizeof(double), s)); return; }
  HiScope hs(a);
  int64_t nb = (n + kGroup - 1) / kGroup;
  double* p = nb == 1 ? d_out : a.hi_n<double>(nb);
  tree_group_kernel<double><<<(unsigned)nb, kRedThreads, 0, s>>>(x, n, p);
  LVG_LAUNCH();
  if (nb > 1) finish_impl(p, nb, d_out, a, s);
}

void tree_sum_f32(const float* x, int64_t n, double* d_out, Arena& a, cudaStream_t s) {
  if (n <= 0) { LVG_CUDA(cudaMemsetAsync(d_out, 0, sizeof(double), s)); return; }
  HiScope hs(a);
  int64_t nb = (n + kGroup - 1) / kGroup;
  double* p = nb == 1 ? d_out : a.hi_n<double>(nb);
  tree_group_kernel<float><<<(unsigned)nb, kRedThreads, 0, s>>>(x, n, p);
  LVG_LAUNCH();
  if (nb > 1) finish_impl(p, nb, d_out, a, s);
}

void tree_finish(const double* partials, int64_t n, double* d_out, Arena& a, cudaStream_t s) {
  if (n <= 1) {
    if (n == 1) LVG_CUDA(cudaMemcpyAsync(d_out, partials, sizeof(double), cudaMemcpyDeviceToDevice, s));
    else LVG_CUDA(cudaMemsetAsync(d_out, 0, sizeof(double), s));
    return;
  }
  finish_impl(partials, n, d_out, a, s);
}

int radix_sort_pairs(uint64_t* k0, float* v0, uint64_t* k1, float* v1, int64_t n, int bits, Arena& a,
                     cudaStream_t s) {
  return radix_sort_range(k0, v0, k1, v1, n, 0, bits, a, s);
}

int radix_sort_range(uint64_t* k0, float* v0, uint64_t* k1, float* v1, int64_t n, int lo, int bits, Arena& a,
                     cudaStream_t s) {
  if (n >= ((int64_t)1 << 32)) throw Error(LVG_ERR_CAPACITY, "radix sort limited to 2^32-1 entries");
  if (lo < 0 || lo >= 64) throw Error(LVG_ERR_INVALID_ARG, "radix sort: first key bit out of range");
  bits = std::min(bits, 64 - lo);
  if (n <= 1 || bits <= 0) return 0;
  static std::once_flag attr_once;
  std::call_once(attr_once, [] {
    LVG_CUDA(cudaFuncSetAttribute(rs_onesweep_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(RsSmem<true>)));
    LVG_CUDA(cudaFuncSetAttribute(rs_onesweep_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(RsSmem<false>)));
  });
  const int npass = (bits + 7) / 8;
  HiScope hs(a);
  const int64_t ntiles = (n + kRsTile - 1) / kRsTile;
  unsigned long long* look = a.hi_n<unsigned long long>(ntiles * kRadix);
  uint32_t* ghist = a.hi_n<uint32_t>(kRsMaxPasses * kRadix + kRsMaxPasses + 1);
  uint32_t* counters = ghist + kRsMaxPasses * kRadix;
  uint32_t* err = counters + kRsMaxPasses;
  LVG_CUDA(cudaMemsetAsync(look, 0, sizeof(unsigned long long) * ntiles * kRadix, s));
  LVG_CUDA(cudaMemsetAsync(ghist, 0, sizeof(uint32_t) * (kRsMaxPasses * kRadix + kRsMaxPasses + 1), s));
  const int64_t ublocks = std::min<int64_t>((n + kRsThreads - 1) / kRsThreads, 148 * 8);
  rs_upfront_kernel<<<(unsigned)ublocks, kRsThreads, 0, s>>>(k0, n, lo, bits, npass, ghist);
  LVG_LAUNCH();
  rs_gscan_kernel<<<1, kRsThreads, 0, s>>>(ghist, npass);
  LVG_LAUNCH();
  int cur = 0;
  uint64_t* K[2] = {k0, k1};
  float* Vv[2] = {v0, v1};
  for (int p = 0; p < npass; ++p) {
    const uint32_t dmask = (1u << std::min(8, bits - 8 * p)) - 1u;
    if (v0)
      rs_onesweep_kernel<true><<<(unsigned)ntiles, kRsThreads, sizeof(RsSmem<true>), s>>>(
          K[cur], Vv[cur], K[cur ^ 1], Vv[cur ^ 1], n, lo + 8 * p, dmask, p, ghist + p * kRadix, look, counters + p,
          err, g_rs_spin_limit.load(), g_rs_hold_tile.load());
    else
      rs_onesweep_kernel<false><<<(unsigned)ntiles, kRsThreads, sizeof(RsSmem<false>), s>>>(
          K[cur], nullptr, K[cur ^ 1], nullptr, n, lo + 8 * p, dmask, p, ghist + p * kRadix, look, counters + p, err,
          g_rs_spin_limit.load(), g_rs_hold_tile.load());
    LVG_LAUNCH();
    cur ^= 1;
  }
  if (fetch_one(err, a, s)) throw Error(LVG_ERR_CUDA, "radix sort look-back did not complete");
  return cur;
}

}  // namespace lvg

extern "C" lvg_status lvg_debug_radix_hold(int32_t spin_limit, int64_t hold_tile) {
  if (spin_limit < 1) return LVG_ERR_INVALID_ARG;
  lvg::g_rs_spin_limit.store(spin_limit);
  lvg::g_rs_hold_tile.store(hold_tile);
  return LVG_OK;
}
