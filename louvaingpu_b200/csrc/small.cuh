// Whole dendrograms of small graphs inside a few launches (small.cu).
#pragma once
#include "louvain.cuh"

namespace lvg {

constexpr int32_t kSmallMaxV = 1 << 18;     // communities of a packed table slot
constexpr int kSmallMaxBlocks = 160;
constexpr int kSmallClusterBlocks = 16;     // a single run's cluster, up to this many entries and vertices;
constexpr int64_t kSmallClusterEntries = 64 * 1024;   // above, a cooperative grid of the whole chip
constexpr int32_t kSmallLevels = 48;        // levels one launch may record
constexpr int32_t kSmallPassCap = 4096;     // passes of a level before it is left to the caller
constexpr int kSmallPhases = 4;             // build, passes, renumbering, coarsening

struct SmallLevel {
  int32_t V, C, passes, pad;
  int64_t E, nnz;
  double q_start, q_level;
  float ticks[kSmallPhases];
  float pass_ticks[2];      // the moves of the first two passes; SmallJob::pass_ticks has any others
  int64_t part_off;         // partition at parts + part_off, labels V later
};

struct SmallResult {
  int32_t n_levels;         // levels finished
  int32_t n_comms;          // communities of the last finished level
  int32_t open;             // 1: the next level was left to the caller, its list as below
  int32_t status;           // lvg_status of the run
  int32_t bad;              // an entry out of range or with a bad weight
  int32_t V;                // list of the last level (or of the open one)
  int32_t buf;              // -1: the job's own list, else coarse list buffer 0 or 1
  int32_t finished;         // 1: the launch came to its end (0: a barrier's wait ran out)
  int64_t E;
  double ms_per_tick;
  double mod;               // Q of the last finished level
  double q_final;           // FP64 modularity of comp over the job's list (want_q)
};

struct SmallOut {
  SmallResult res;
  SmallLevel lv[kSmallLevels];
};

// One graph (or the rest of a run from a coarse level on).
struct SmallJob {
  const int32_t* src;
  const int32_t* dst;
  const float* w;
  int64_t E;
  int32_t V;
  int32_t level0;           // level of the given list in its run
  double mod;               // Q of the level before (level0 > 0)
  char* lists;              // two coarse list buffers of E entries each
  char* work;               // small_work_bytes(V, E, dbl, blocks)
  int32_t* parts;           // per-level partitions and labels, the first level's last, or nullptr
  int64_t parts_cap;        // ints
  int32_t* comp;            // [V] composition of the levels' partitions
  double* state;            // small_state_bytes(V), or nullptr: the state the run ends in, over the last
                            // level's communities: tot, in, then (int32) sizes, one array behind the other
  SmallResult* res;
  SmallLevel* lv;           // [kSmallLevels], or nullptr
  float* pass_ticks;        // [kSmallPassCap] moves of the last level's passes from the third on, or nullptr
  int32_t check;            // 1: ids, weights, order and symmetry not checked yet
  int32_t want_q;
  int32_t dbl;              // 1: work has room for lists in any order (small_work_bytes with dbl)
  int32_t blocks;           // most blocks that work on it at a time
};

struct SmallCfg {
  double pass_min, level_min;
  int32_t max_passes, max_levels;
  int32_t hold = -1;                // grid: a block that stays away (test hook)
  int64_t wait_ns = 4000000000ll;   // limit of a grid barrier's wait
};

size_t small_list_bytes(int64_t E);           // both coarse list buffers
size_t small_work_bytes(int32_t V, int64_t E, bool dbl, int blocks);
inline size_t small_state_bytes(int32_t V) { return (2 * sizeof(double) + sizeof(int32_t)) * (size_t)V; }
// Coarse list buffer `buf` of a job's lists.
void small_list(char* lists, int64_t E, int buf, int32_t** src, int32_t** dst, float** w);
// True when the sizes are ones this path takes.
bool small_fits(int64_t V, int64_t E, int64_t max_entries);
// Runs n jobs (device array), each by a cluster of K blocks.  The caller has
// cleared the results (finished == 0).  False: the device, or the part of it
// the stream may use, does not take such a launch; nothing has run.
bool small_run(const SmallJob* d_jobs, int n, int K, const SmallCfg& cfg, cudaStream_t s);
// Runs one job (work: its work area) by a cooperative grid of
// K <= small_grid_blocks() blocks.  False: as small_run's.
bool small_run_grid(const SmallJob* d_job, void* work, int K, const SmallCfg& cfg, cudaStream_t s);
int small_grid_blocks();

}  // namespace lvg
